// resident.cu -- resident CG and BiCGSTAB (resident.cuh).
//
// What bounds a small or middling solve launched kernel by kernel is not the
// matrix but the three to seven dependent launches of an iteration: each starts
// cold, drains, and ends in a chain of L2 round trips (partial sums, ticket, the
// last CTA's total).  Here one cooperative launch holds a CTA on every SM for the
// whole solve:
//   * a CTA owns a run of slices (32 block rows each); x, r, p, ... of its rows lie in
//     its shared memory, as many of them as fit beside the ring (`near`; in the order of
//     their use, the inverse diagonal blocks last), the others in global scratch that
//     only it reads.  With block Jacobi, 3x3 blocks and 152 SMs all fit up to 53,500 block
//     rows (FP64 CG), 34,000 (FP64 BiCGSTAB), 68,000 (mixed CG), 53,500 (mixed BiCGSTAB); at
//     119,000 rows two of FP64 CG's six, above 185,000 none;
//   * only the vector that the next product gathers is written to global memory;
//   * the CTA's slots are cut into 16 equal runs, one per warp, whatever the
//     slices' boundaries: a warp stores the sums of each slice it touches and a
//     row adds its few segments in a fixed order;
//   * each warp streams its run through a ring of shared-memory stages (bulk
//     copies); the ring runs on into the next product, so it fills while the
//     CTAs wait for one another, and a run that fits the ring is loaded once;
//   * the grid-wide sums are exchanges: every CTA writes its partial into every
//     other's inbox and adds its own inbox in CTA order, so every CTA holds the same
//     bits and takes the same decisions; an exchange is also the grid's barrier.
//     (Inboxes: 152 CTAs that all poll the same 152 slots take 7,600-9,600 cycles
//     per exchange, a counter 4,800, inboxes 3,700, or 5,600 with the fences that
//     publish a vector.)
//   * scalars are formed by one thread while the others wait: on GB300 an FP64
//     division takes 660 cycles in one warp and 2,560 in sixteen.
// An FP64 iteration has three exchanges (CG) or five (BiCGSTAB); FP32 CG forms
// p = z + beta p inside the gather and has two.  In FP64 that would add a third
// to the work of GB300's slow FP64 pipe (two multiply-adds per clock and SM),
// more than the exchange costs.
// Measured, us per iteration, kernel by kernel -> resident, block rows of cubes of
// hexes (block Jacobi):
//              2,197        9,261        24,389       50,653       91,125       148,877
//   CG FP64    35.5 -> 13.7 43.4 -> 16.4 54.3 -> 23.9 61.0 -> 38.8 72.1 -> 60.9 94.4 -> 90.5
//   CG mixed   21.3 ->  9.0 21.2 ->  9.6 20.3 -> 11.9 22.3 -> 15.8 30.9 -> 24.6 32.7 -> 45.8
//   BiCG FP64  61.4 -> 25.1 72.6 -> 31.3 91.7 -> 45.2  107 -> 75.0  138 ->  121  180 ->  181
//   BiCG mixed 48.2 -> 18.7 46.2 -> 20.2 44.5 -> 24.4 48.0 -> 31.0 66.9 -> 52.6 75.3 -> 94.4
// (mixed, kernel by kernel, reads the upper half of the matrix from HBM; resident
// reads the whole FP32 copy, which pays while that fits L2: 98 MB at 91,125 rows).  Other
// kinds of rows and the limits: krylov.cu, resident_pays.
//
// Every wait is bounded: a CTA whose inbox does not fill within the limit raises
// `err` and leaves, and so do the others; copies in flight are waited for first.
#include <algorithm>
#include <cmath>

#include "bulk.cuh"
#include "resident.cuh"

namespace pfg {
namespace {

constexpr int kNT = 512;  // threads per CTA, one CTA per SM
constexpr int kNW = kNT / 32;
constexpr uint64_t kWaitNs = 4000000000ull;
constexpr size_t kSmemMax = 222 * 1024;  // dynamic shared memory (227 KB less the static part)
constexpr int kMaxStages = 8;
// Mixed solves: replacements in a row without a 10 % fall of the FP64 residual,
// and rejected FP32 passes in a row, before FP64 takes over (as run_mixed).
constexpr int kStallCG = 4, kStallBiCG = 8, kReject = 2;

__device__ __forceinline__ double empty_slot() { return __longlong_as_double(-1ll); }
__device__ __forceinline__ bool is_empty(double v) { return __double_as_longlong(v) == -1ll; }

// An exchange entry: kResValues doubles, each valid once it is not the empty
// slot (so the pair need not travel as one).
template <int NV>
__device__ __forceinline__ void st_entry(double *p, double a, double b)
{
    if (NV == 2)
        asm volatile("st.volatile.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(a), "d"(b) : "memory");
    else
        asm volatile("st.volatile.global.f64 [%0], %1;" ::"l"(p), "d"(a) : "memory");
}
template <int NV>
__device__ __forceinline__ void ld_entry(const double *p, double &a, double &b)
{
    if (NV == 2)
        asm volatile("ld.volatile.global.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "l"(p) : "memory");
    else
        asm volatile("ld.volatile.global.f64 %0, [%1];" : "=d"(a) : "l"(p) : "memory");
}

enum Step { kGo, kDone, kReplace, kLost };

// The scalars an iteration changes.
struct Live {
    double beta, rho, inv_rho, alpha, c2, c3, rr;  // rho: <r, z> (CG) or c1 = <r0, r> (BiCGSTAB)
    double goal, goal1, near0;                     // squared: tol |b|, and tol sqrt(rr1) and er0 (reference stop rule)
    double bb, rr1;
    int exact;                                     // a square is no measure: negative, or lost to underflow
    float beta32, alpha32, c3_32;                  // what the FP32 row passes read
    float rmax, rmin;
    int iter, parity, status, breakdowns, poisoned, next;
};

struct ResShared {
    double red[kResValues][kNW];
    float redf[2 * kResValues][kNW];
    double tot[2][kResValues];
    ResState state;
    Live live;
    int fail;
};

// The CTA's place in the grid and its exchanges.
struct Grid {
    ResShared *sh;
    double *slots;
    int *err;
    int s0, nsl, lane, wid;
    unsigned round;

    // the entry of CTA `from` in CTA `to`'s inbox
    __device__ double *entry(unsigned buf, int to, int from) const
    {
        return slots + (((size_t)buf * kResMaxCtas + to) * kResMaxCtas + from) * kResValues;
    }

    // v (valid in warp 0) -> the grid's totals in every thread; `fin(totals)` runs
    // in one thread before the others go on, `mid()` in all threads while the
    // values travel.  PUBLISH: what the CTA wrote to global memory before is
    // visible to every CTA after.  Buffers rotate over kResRounds rounds; a CTA
    // empties its inbox of the buffer four rounds ahead, which it has read (it was
    // used four rounds ago) and which a published round orders before its next use
    // (no loop here goes four rounds without one).  False: a wait ran out.
    // SUM false: a barrier only, without the 650 cycles of the additions.
    template <int NV, bool PUBLISH, bool SUM = true, typename Mid, typename Fin>
    __device__ bool exchange(double (&v)[NV], const Mid &mid, const Fin &fin)
    {
        const unsigned buf = round % kResRounds;
        const int G = gridDim.x;
        if (wid == 1) {
            const unsigned ahead = (round + kResRounds / 2) % kResRounds;
            for (int c = lane; c < G; c += 32) st_entry<2>(entry(ahead, blockIdx.x, c), empty_slot(), empty_slot());
        }
        if (wid == 0) {
            if (PUBLISH) __threadfence();
#pragma unroll
            for (int k = 0; k < NV; ++k)
                if (v[k] != v[k]) v[k] = __longlong_as_double(0x7ff8000000000000ll);  // a NaN that is not the empty slot
            for (int c = lane; c < G; c += 32) st_entry<NV>(entry(buf, c, blockIdx.x), v[0], v[NV - 1]);
        }
        mid();
        if (wid == 0) {
            constexpr int U = kResMaxCtas / 32;
            double t[U][NV];
            bool ok = true;
            uint64_t since = 0;
            for (unsigned spin = 1;; ++spin) {
                bool wait = false;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int c = 32 * u + lane;
                    t[u][0] = t[u][NV - 1] = 0.0;
                    if (c < G) ld_entry<NV>(entry(buf, blockIdx.x, c), t[u][0], t[u][NV - 1]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int k = 0; k < NV; ++k) wait |= is_empty(t[u][k]);
                if (!__any_sync(0xffffffffu, wait)) break;
                if ((spin & 1023u) == 0) {
                    const uint64_t now = global_ns();
                    if (since == 0) since = now;
                    const bool stop = now - since > kWaitNs || *(volatile int *)err != 0;
                    if (__any_sync(0xffffffffu, stop)) {
                        ok = false;
                        break;
                    }
                }
            }
            if (PUBLISH) __threadfence();
            static_assert(U == 5, "the sum below takes five values per lane");
            double acc[NV];
            if (SUM) {
#pragma unroll
                for (int k = 0; k < NV; ++k) acc[k] = ((t[0][k] + t[1][k]) + (t[2][k] + t[3][k])) + t[4][k];
                const double all = lanes_sum<NV>(acc, lane);
#pragma unroll
                for (int k = 0; k < NV; ++k) acc[k] = __shfl_sync(0xffffffffu, all, 16 * k);
            }
            if (lane == 0) {
                if (!ok) {
                    sh->fail = 1;
                    *(volatile int *)err = 1;
                }
                if (SUM) {
#pragma unroll
                    for (int k = 0; k < NV; ++k) sh->tot[round & 1][k] = acc[k];
                    fin(acc);
                }
            }
        }
        __syncthreads();
        if (SUM)
#pragma unroll
            for (int k = 0; k < NV; ++k) v[k] = sh->tot[round & 1][k];
        ++round;
        return sh->fail == 0;
    }

    __device__ int active() const { return min(kNW, nsl); }  // warps that own rows

    template <int NV, bool PUBLISH, typename Mid, typename Fin>
    __device__ bool sum(double (&v)[NV], const Mid &mid, const Fin &fin)
    {
        const int act = active();
        if (wid < act) {
            const double t = lanes_sum<NV>(v, lane);
            if (NV == 1 ? lane == 0 : (lane & 15) == 0) sh->red[lane >> 4][wid] = t;
        }
        __syncthreads();
        if (wid == 0) {
            // lane 16 k + w: value k of warp w
            double t = (lane & 15) < act && lane < 16 * NV ? sh->red[NV == 1 ? 0 : lane >> 4][lane & 15] : 0.0;
            for (int o = 1; o < act; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
#pragma unroll
            for (int k = 0; k < NV; ++k) v[k] = __shfl_sync(0xffffffffu, t, 16 * k);
        }
        return exchange<NV, PUBLISH>(v, mid, fin);
    }

    __device__ static void merge(Comp32 &t)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float s2 = __shfl_xor_sync(0xffffffffu, t.s, o);
            const float c2 = __shfl_xor_sync(0xffffffffu, t.c, o);
            comp_merge(t, s2, c2);
        }
    }
    // compensated FP32 sums: the CTA's pair becomes a double, the CTAs' are added in FP64
    template <int NV, bool PUBLISH, typename Mid, typename Fin>
    __device__ bool sum(Comp32 (&v)[NV], const Mid &mid, const Fin &fin)
    {
        const int act = active();
        if (wid < act) {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                merge(v[k]);
                if (lane == 0) {
                    sh->redf[2 * k][wid] = v[k].s;
                    sh->redf[2 * k + 1][wid] = v[k].c;
                }
            }
        }
        __syncthreads();
        double tot[NV];
        if (wid == 0)
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                Comp32 t{lane < act ? sh->redf[2 * k][lane] : 0.f, lane < act ? sh->redf[2 * k + 1][lane] : 0.f};
                if (act > 1) merge(t);
                tot[k] = __shfl_sync(0xffffffffu, (double)t.s + (double)t.c, 0);
            }
        return exchange<NV, PUBLISH>(tot, mid, fin);
    }
    __device__ bool barrier()
    {
        double v[1] = {0.0};
        __syncthreads();
        return exchange<1, true, false>(v, [] {}, [](double(&)[1]) {});
    }
};

template <typename T>
struct Dot;
template <>
struct Dot<double> {
    using type = double;
    __device__ static double zero() { return 0.0; }
    __device__ static void add(double &a, double x, double y) { a = fma(x, y, a); }
};
template <>
struct Dot<float> {
    using type = Comp32;
    __device__ static Comp32 zero() { return Comp32{0.f, 0.f}; }
    __device__ static void add(Comp32 &a, float x, float y) { comp_add_prod(a, x, y); }
};

// A CTA's slots (those of its slices, in order) cut into kNW runs, equal but for
// one slot, empty runs last.  A run and a slice that meet make a segment; the
// segment of warp w and slice sl has the index sl + w (the next one in slot order
// has a larger sl, w or both), and a slice's segments are those of consecutive warps.
struct Cut {
    const int64_t *sp;  // sptr of the CTA's slices (shared memory)
    int nsl;
    __device__ int slots() const { return (int)(sp[nsl] - sp[0]); }
    __device__ int start(int w) const
    {
        const int n = slots();
        return n / kNW * w + min(w, n % kNW);
    }
    // the warp whose run holds slot t (t < slots())
    __device__ int warp_of(int t) const
    {
        const int n = slots(), q = n / kNW, rem = n % kNW, big = rem * (q + 1);
        return t < big ? t / (q + 1) : rem + (t - big) / q;
    }
};

// slots per ring stage
template <typename T>
constexpr int kChunk = sizeof(T) == 8 ? 1 : 4;

template <int BS, typename T>
constexpr int kStageBytes = kChunk<T> * 32 * (4 + BS * BS * (int)sizeof(T));

// A warp's run of slots streamed through its ring, product after product.  The
// chunks of a run (kChunk slots, cut at slice boundaries) are produced and
// consumed in order, cyclically; when the whole run fits the ring it is loaded
// once and stays.
template <int BS, typename T>
struct Stream {
    static constexpr int CH = kChunk<T>;
    SellView<T> A;
    const int64_t *sp;
    uint64_t *bar;
    unsigned char *ring;
    int nst, lane, t0, t1, sl0;  // slots [t0, t1) of the CTA's, the first in slice sl0
    int chunks;                  // of the run
    bool stays;
    int pt, psl, pst, cst, flying;
    unsigned cph;

    __device__ void init(const SellView<T> &a, const Cut &cut, uint64_t *bars, unsigned char *stages, int n)
    {
        A = a;
        sp = cut.sp;
        lane = threadIdx.x & 31;
        const int wid = threadIdx.x >> 5;
        nst = n;
        bar = bars + wid * nst;
        ring = stages + (size_t)wid * nst * kStageBytes<BS, T>;
        if (lane == 0) {
            for (int i = 0; i < nst; ++i) mbar_init(bar + i, 1);
            fence_proxy_async_smem();
        }
        __syncwarp();
        t0 = cut.start(wid);
        t1 = cut.start(wid + 1);
        sl0 = 0;
        while (sl0 < cut.nsl && (int)(sp[sl0 + 1] - sp[0]) <= t0) ++sl0;
        chunks = 0;
        for (int t = t0, sl = sl0; t < t1; ++chunks) t += next(t, sl);
        stays = chunks <= nst;
        pt = t0;
        psl = sl0;
        pst = cst = flying = 0;
        cph = 0;
        const int fill = min(chunks, nst);
        for (int i = 0; i < fill; ++i) produce();
    }
    // slots of the chunk at t in slice sl (advanced past finished slices by the caller's t)
    __device__ int next(int t, int &sl) const
    {
        while ((int)(sp[sl + 1] - sp[0]) <= t) ++sl;
        return min(CH, min(t1, (int)(sp[sl + 1] - sp[0])) - t);
    }
    __device__ void produce()
    {
        const int n = next(pt, psl);
        if (lane == 0) {
            unsigned char *dst = ring + (size_t)pst * kStageBytes<BS, T>;
            const int64_t at = sp[0] + pt;
            mbar_arrive_expect_tx(bar + pst, (unsigned)(n * 32 * (4 + BS * BS * (int)sizeof(T))));
            bulk_g2s(dst, A.col + at * 32, (unsigned)(n * 128), bar + pst);
            bulk_g2s(dst + CH * 128, A.val + at * 32 * (BS * BS), (unsigned)(n * 32 * BS * BS * (int)sizeof(T)),
                     bar + pst);
        }
        pst = pst + 1 == nst ? 0 : pst + 1;
        ++flying;
        pt += n;
        if (pt >= t1) {
            pt = t0;
            psl = sl0;
        }
    }
    // buf[((sl + warp) * BS + i) * 32 + lane] = the segment's sums; false: a copy did not arrive
    template <typename Src>
    __device__ bool apply(const Src &src, T *buf)
    {
        if (chunks == 0) return true;
        const int wid = threadIdx.x >> 5;
        int sl = sl0;
        int t = t0, n = next(t, sl);
        int st = stays ? 0 : cst;
        unsigned ph = stays ? 0u : cph;
        T xv[CH][BS];
        if (!__all_sync(0xffffffffu, mbar_wait(bar + st, ph))) return false;
        const unsigned char *stage = ring + (size_t)st * kStageBytes<BS, T>;
#pragma unroll
        for (int j = 0; j < CH; ++j)
            if (j < n) src(reinterpret_cast<const int *>(stage)[j * 32 + lane], xv[j]);
        T y[BS];
#pragma unroll
        for (int r = 0; r < BS; ++r) y[r] = T(0);
        for (int i = 0; i < chunks; ++i) {
            // the next chunk's gathers go out before this one's products
            const int tn = t + n;
            int sn = sl, nn = 0, stn = st + 1;
            unsigned phn = ph;
            T xn[CH][BS];
            const unsigned char *stage_n = stage;
            if (stn == nst) {
                stn = 0;
                phn ^= 1u;
            }
            if (i + 1 < chunks) {
                nn = next(tn, sn);
                if (!__all_sync(0xffffffffu, mbar_wait(bar + stn, phn))) return false;
                stage_n = ring + (size_t)stn * kStageBytes<BS, T>;
#pragma unroll
                for (int j = 0; j < CH; ++j)
                    if (j < nn) src(reinterpret_cast<const int *>(stage_n)[j * 32 + lane], xn[j]);
            }
            const T *vs = reinterpret_cast<const T *>(stage + CH * 128);
#pragma unroll
            for (int j = 0; j < CH; ++j)
                if (j < n)
#pragma unroll
                    for (int r = 0; r < BS; ++r)
#pragma unroll
                        for (int c = 0; c < BS; ++c)
                            y[r] = fma(vs[(j * BS * BS + r * BS + c) * 32 + lane], xv[j][c], y[r]);
            if (!stays) {  // every lane has read the stage: refill it
                __syncwarp();
                if (lane == 0) fence_proxy_async_smem();
                --flying;
                produce();
            }
            if (sn != sl || nn == 0) {  // the slice's last chunk of this run
#pragma unroll
                for (int r = 0; r < BS; ++r) {
                    buf[((sl + wid) * BS + r) * 32 + lane] = y[r];
                    y[r] = T(0);
                }
            }
            t = tn;
            n = nn;
            sl = sn;
            st = stn;
            ph = phn;
            stage = stage_n;
#pragma unroll
            for (int j = 0; j < CH; ++j)
#pragma unroll
                for (int r = 0; r < BS; ++r) xv[j][r] = xn[j][r];
        }
        if (!stays) {
            cst = st;
            cph = ph;
        }
        return true;
    }
    // waits (bounded) for the copies in flight
    __device__ void drain()
    {
        int st = stays ? 0 : cst;
        unsigned ph = stays ? 0u : cph;
        for (int i = 0; i < flying; ++i) {
            (void)mbar_wait(bar + st, ph);
            if (++st == nst) {
                st = 0;
                ph ^= 1u;
            }
        }
    }
};

// The same product without a ring (the FP64 residuals of a mixed solve).
template <int BS, typename Src>
__device__ void apply_plain(const SellView<double> &A, const Cut &cut, const Src &src, double *buf)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int t1 = cut.start(wid + 1);
    int t = cut.start(wid), sl = 0;
    const int64_t first = cut.sp[0];
    while (t < t1) {
        while ((int)(cut.sp[sl + 1] - first) <= t) ++sl;
        const int e = min(t1, (int)(cut.sp[sl + 1] - first));
        double y[BS];
#pragma unroll
        for (int r = 0; r < BS; ++r) y[r] = 0.0;
#pragma unroll 2
        for (; t < e; ++t) {
            const int64_t at = first + t;
            double av[BS * BS], xv[BS];
            const int c = ld_stream(A.col + at * 32 + lane);
#pragma unroll
            for (int k = 0; k < BS * BS; ++k) av[k] = ld_stream(A.val + (at * (BS * BS) + k) * 32 + lane);
            src(c, xv);
#pragma unroll
            for (int r = 0; r < BS; ++r)
#pragma unroll
                for (int k = 0; k < BS; ++k) y[r] = fma(av[r * BS + k], xv[k], y[r]);
        }
#pragma unroll
        for (int r = 0; r < BS; ++r) buf[((sl + wid) * BS + r) * 32 + lane] = y[r];
    }
}

// The rows a thread updates: slice sl, row (s0 + sl) * 32 + lane.
#define RES_ROWS(g, nbrows)                                              \
    for (int sl = (g).wid; sl < (g).nsl; sl += kNW)                      \
        if (const int64_t row = ((int64_t)(g).s0 + sl) * 32 + (g).lane; row < (nbrows))

constexpr unsigned char kNoSegment = 255;  // a slice without slots

// A published vector has 4 entries per row of a 3x3-block system (one or two
// 16-byte loads per gathered row instead of three strided ones), else 1.
template <int BS>
constexpr int kPub = BS == 3 ? 4 : BS;

template <int BS>
__device__ __forceinline__ void gather(const float *v, int64_t row, float (&x)[BS])
{
    if (BS == 3) {
        const float4 q = *reinterpret_cast<const float4 *>(v + 4 * row);
        x[0] = q.x;
        x[BS > 1 ? 1 : 0] = q.y;
        x[BS > 2 ? 2 : 0] = q.z;
        if (BS == 1) x[0] = q.x;
    } else {
        x[0] = v[row];
    }
}
template <int BS>
__device__ __forceinline__ void gather(const double *v, int64_t row, double (&x)[BS])
{
    if (BS == 3) {
        const double2 q = *reinterpret_cast<const double2 *>(v + 4 * row);
        x[0] = q.x;
        x[BS > 1 ? 1 : 0] = q.y;
        x[BS > 2 ? 2 : 0] = v[4 * row + 2];
        if (BS == 1) x[0] = q.x;
    } else {
        x[0] = v[row];
    }
}
template <int BS>
__device__ __forceinline__ void publish(float *v, int64_t row, const float (&x)[BS])
{
    if (BS == 3)
        *reinterpret_cast<float4 *>(v + 4 * row) = make_float4(x[0], x[BS > 1 ? 1 : 0], x[BS > 2 ? 2 : 0], 0.f);
    else
        v[row] = x[0];
}
template <int BS>
__device__ __forceinline__ void publish(double *v, int64_t row, const double (&x)[BS])
{
    if (BS == 3) {
        *reinterpret_cast<double2 *>(v + 4 * row) = make_double2(x[0], x[BS > 1 ? 1 : 0]);
        v[4 * row + 2] = x[BS > 2 ? 2 : 0];
    } else {
        v[row] = x[0];
    }
}

// A CTA's share of one solve in precision T.  Own vectors: [slice][component][lane].
template <int BS, typename T>
struct Solve {
    Grid *g;
    Stream<BS, T> mat;
    const unsigned char *wlo, *whi;  // warps whose segments make up a slice
    int64_t nb;
    const T *dinv;  // own planes of the inverse diagonal blocks, null: no preconditioner
    T *buf;

    __device__ int own(int sl, int i) const { return (sl * BS + i) * 32 + g->lane; }
    // sum of a row's segments, kept in the first one's place
    __device__ void collect(int sl, T (&q)[BS]) const
    {
        const int lo = wlo[sl], hi = whi[sl];
        T *b0 = buf + (sl + lo) * BS * 32 + g->lane;
        if (hi == kNoSegment) {
#pragma unroll
            for (int i = 0; i < BS; ++i) b0[i * 32] = q[i] = T(0);
            return;
        }
#pragma unroll
        for (int i = 0; i < BS; ++i) q[i] = b0[i * 32];
        if (hi == lo) return;
        const T *bw = b0;
        for (int w = lo; w < hi; w += 4) {  // four segments' loads at once
            T t[4][BS];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < BS; ++i) t[u][i] = w + u < hi ? bw[((u + 1) * BS + i) * 32] : T(0);
#pragma unroll
            for (int i = 0; i < BS; ++i) q[i] += (t[0][i] + t[1][i]) + (t[2][i] + t[3][i]);
            bw += 4 * BS * 32;
        }
#pragma unroll
        for (int i = 0; i < BS; ++i) b0[i * 32] = q[i];
    }
    __device__ T collected(int sl, int i) const { return buf[((sl + wlo[sl]) * BS + i) * 32 + g->lane]; }
    __device__ void keep(int sl, int i, T v) const { buf[((sl + wlo[sl]) * BS + i) * 32 + g->lane] = v; }
    __device__ void precond(int sl, const T (&r)[BS], T (&z)[BS]) const
    {
        if (dinv == nullptr) {
#pragma unroll
            for (int i = 0; i < BS; ++i) z[i] = r[i];
            return;
        }
        const T *D = dinv + sl * (BS * BS * 32) + g->lane;
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            T s = T(0);
#pragma unroll
            for (int j = 0; j < BS; ++j) s = fma(D[(i * BS + j) * 32], r[j], s);
            z[i] = s;
        }
    }
    template <typename Src>
    __device__ void product(const Src &src)
    {
        if (!mat.apply(src, buf)) {
            g->sh->fail = 1;
            *(volatile int *)g->err = 1;
        }
        __syncthreads();
    }
};

// (integer test: an FP64 comparison costs 65 cycles)
__device__ __forceinline__ bool finite(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

// a / b by way of the reciprocal that was formed meanwhile, unless that is out of range (b of
// a right-hand side of 1e-153, say)
__device__ __forceinline__ double quotient(double a, double b, double inv_b)
{
    const int e = __double2hiint(inv_b) & 0x7ff00000;
    return e != 0 && e != 0x7ff00000 ? a * inv_b : a / b;
}

// Whether the square of a limit can stand for it: a division or square root takes
// 660 cycles of an iteration's serial part, a comparison 65.
__device__ __forceinline__ bool square_holds(double limit, double square)
{
    return limit == 0.0 || (limit > 0.0 && square > 1e-280);
}

// FP64: the stop test on the recursive residual (reference rule: FEMSolverClass.f90:2275-2289)
template <bool REFERENCE>
__device__ __forceinline__ bool reached(const Live &v, const ResArgs &a, double rr)
{
    if (v.exact)
        return REFERENCE ? sqrt(rr / v.rr1) < a.tol || sqrt(rr) < a.er0 : sqrt(rr) <= a.tol * sqrt(v.bb);
    return REFERENCE ? rr < v.goal1 || rr < v.near0 : rr <= v.goal;
}

// FP32: what an iteration's end asks for (replace on progress, at the tolerance,
// or when the recursion diverged)
__device__ __forceinline__ bool replace_due(Live &v, const ResArgs &a, double rr)
{
    const float rn = sqrtf((float)rr);
    v.rmax = fmaxf(v.rmax, rn);
    v.rmin = fminf(v.rmin, rn);
    return rn < (float)a.delta * v.rmax || (double)rn * (double)rn <= v.goal || rn > 1000.f * v.rmin;
}

// One CG iteration.  FP64: p is published, three exchanges.  FP32: z and the
// previous p are published and p = z + beta p is formed in the gather, two.
template <int BS, typename T>
__device__ Step cg_step(Solve<BS, T> &S, const ResArgs &a, T *xs, T *rs, T *ps, T *zs, T *pg, T *zg, T *pA, T *pB)
{
    constexpr bool f64 = sizeof(T) == 8;
    Grid &g = *S.g;
    Live &v = g.sh->live;
    const T beta = f64 ? (T)0 : (T)v.beta32;
    const int par = v.parity;
    const T *pold = par ? pB : pA;
    T *pnew = par ? pA : pB;
    if (f64)
        S.product([&](int c, T(&x)[BS]) {
            gather<BS>(pg, c, x);
        });
    else
        S.product([&](int c, T(&x)[BS]) {
            T z[BS];
            gather<BS>(pold, c, x);
            gather<BS>(zg, c, z);
#pragma unroll
            for (int i = 0; i < BS; ++i) x[i] = fma(beta, x[i], z[i]);
        });
    typename Dot<T>::type d1[1] = {Dot<T>::zero()};
    RES_ROWS(g, S.nb)
    {
        T q[BS], p[BS];
        S.collect(sl, q);
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            p[i] = ps[S.own(sl, i)];
            if (!f64) ps[S.own(sl, i)] = p[i] = fma(beta, p[i], zs[S.own(sl, i)]);
            Dot<T>::add(d1[0], p[i], q[i]);
        }
        if (!f64) publish<BS>(pnew, row, p);
    }
    if (!g.template sum<1, false>(d1, [] {}, [&](double(&t)[1]) {
            const double pq = f64 ? t[0] : (double)(float)t[0];
            v.next = kGo;
            if (!(pq > 0.0) || !finite(pq)) {
                v.status = PFG_E_BREAKDOWN;
                v.next = kDone;
            } else if (f64) {
                v.alpha = v.rho / pq;
            } else {
                v.alpha32 = (float)v.rho / (float)pq;
            }
        }))
        return kLost;
    if (v.next == kDone) return kDone;
    const T alpha = f64 ? (T)v.alpha : (T)v.alpha32;
    if (threadIdx.x == kNT - 1) v.inv_rho = 1.0 / v.rho;
    typename Dot<T>::type d2[2] = {Dot<T>::zero(), Dot<T>::zero()};
    RES_ROWS(g, S.nb)
    {
        T r[BS], z[BS];
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            const int o = S.own(sl, i);
            r[i] = fma(-alpha, S.collected(sl, i), rs[o]);
            rs[o] = r[i];
        }
        S.precond(sl, r, z);
        if (!f64) publish<BS>(zg, row, z);
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            if (f64)
                S.keep(sl, i, z[i]);
            else
                zs[S.own(sl, i)] = z[i];
            Dot<T>::add(d2[0], r[i], z[i]);
            Dot<T>::add(d2[1], r[i], r[i]);
        }
    }
    auto advance_x = [&] {  // while the sums travel
        RES_ROWS(g, S.nb)
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            const int o = S.own(sl, i);
            xs[o] = fma(alpha, ps[o], xs[o]);
        }
    };
    if (!g.template sum<2, !f64>(d2, advance_x, [&](double(&t)[2]) {
            const double rho = f64 ? t[0] : (double)(float)t[0], rr = f64 ? t[1] : (double)(float)t[1];
            v.iter += 1;
            v.parity ^= 1;
            v.next = kGo;
            if (!finite(rho) || !finite(rr)) {
                if (f64) {
                    v.status = PFG_E_NONFINITE;
                    v.next = kDone;
                } else {
                    v.breakdowns += 1;
                    v.poisoned = 1;
                    v.next = kReplace;
                }
                return;
            }
            v.rr = rr;
            if (f64) {
                v.beta = quotient(rho, v.rho, v.inv_rho);
                v.rho = rho;
                if (reached<false>(v, a, rr)) v.next = kDone;
            } else if (replace_due(v, a, rr)) {
                v.next = kReplace;
            } else {
                v.beta32 = (float)(rho * v.inv_rho);
                v.rho = rho;
            }
            if (v.iter >= a.itrmax && v.next != kDone) {
                v.status = PFG_W_NOT_CONVERGED;
                v.next = kDone;
            }
        }))
        return kLost;
    const Step next = (Step)v.next;
    if (f64 && next == kGo) {
        const T bt = (T)v.beta;
        RES_ROWS(g, S.nb)
        {
            T p[BS];
#pragma unroll
            for (int i = 0; i < BS; ++i) {
                const int o = S.own(sl, i);
                ps[o] = p[i] = fma(bt, ps[o], S.collected(sl, i));
            }
            publish<BS>(pg, row, p);
        }
        if (!g.barrier()) return kLost;
    }
    return next;
}

// One BiCGSTAB iteration (bicgstab_CRS_2's loop body with right preconditioning):
// phg and ehg are the published M^-1 p and M^-1 e.
template <int BS, typename T>
__device__ Step bicg_step(Solve<BS, T> &S, const ResArgs &a, T *xs, T *rs, T *r0s, T *ps, T *ys, T *phs, T *ehs,
                          T *phg, T *ehg)
{
    constexpr bool f64 = sizeof(T) == 8;
    Grid &g = *S.g;
    Live &v = g.sh->live;
    // FP64 breakdown ends the solve; an FP32 one asks for a replacement
    auto breakdown = [&]() {
        if (f64) {
            v.status = PFG_E_BREAKDOWN;
            v.next = kDone;
        } else {
            v.breakdowns += 1;
            v.next = kReplace;
        }
    };
    {
        const T beta = f64 ? (T)v.beta : (T)v.beta32, c3 = f64 ? (T)v.c3 : (T)v.c3_32;
        RES_ROWS(g, S.nb)
        {
            T p[BS], h[BS];
#pragma unroll
            for (int i = 0; i < BS; ++i) {
                const int o = S.own(sl, i);
                p[i] = fma(beta, fma(-c3, ys[o], ps[o]), rs[o]);
                ps[o] = p[i];
            }
            S.precond(sl, p, h);
            publish<BS>(phg, row, h);
#pragma unroll
            for (int i = 0; i < BS; ++i) phs[S.own(sl, i)] = h[i];
        }
        if (!g.barrier()) return kLost;
    }
    S.product([&](int c, T(&x)[BS]) { gather<BS>(phg, c, x); });
    typename Dot<T>::type d1[1] = {Dot<T>::zero()};
    RES_ROWS(g, S.nb)
    {
        T q[BS];
        S.collect(sl, q);
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            ys[S.own(sl, i)] = q[i];
            Dot<T>::add(d1[0], r0s[S.own(sl, i)], q[i]);
        }
    }
    if (!g.template sum<1, false>(d1, [] {}, [&](double(&t)[1]) {
            const double c2 = f64 ? t[0] : (double)(float)t[0];
            v.next = kGo;
            if (c2 == 0.0 || !finite(c2)) {
                breakdown();
                return;
            }
            v.c2 = c2;
            if (f64)
                v.alpha = v.rho / c2;
            else
                v.alpha32 = (float)v.rho / (float)c2;
        }))
        return kLost;
    if (v.next != kGo) return (Step)v.next;
    const T alpha = f64 ? (T)v.alpha : (T)v.alpha32;
    RES_ROWS(g, S.nb)
    {
        T e[BS], h[BS];
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            const int o = S.own(sl, i);
            e[i] = fma(-alpha, ys[o], rs[o]);
            rs[o] = e[i];  // e takes r's place until r = e - c3 v
        }
        S.precond(sl, e, h);
        publish<BS>(ehg, row, h);
#pragma unroll
        for (int i = 0; i < BS; ++i) ehs[S.own(sl, i)] = h[i];
    }
    if (!g.barrier()) return kLost;
    S.product([&](int c, T(&x)[BS]) { gather<BS>(ehg, c, x); });
    typename Dot<T>::type d2[2] = {Dot<T>::zero(), Dot<T>::zero()};
    RES_ROWS(g, S.nb)
    {
        T w[BS];
        S.collect(sl, w);
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            Dot<T>::add(d2[0], rs[S.own(sl, i)], w[i]);
            Dot<T>::add(d2[1], w[i], w[i]);
        }
    }
    if (!g.template sum<2, false>(d2, [] {}, [&](double(&t)[2]) {
            const double ev = f64 ? t[0] : (double)(float)t[0], vv = f64 ? t[1] : (double)(float)t[1];
            v.next = kGo;
            if (vv == 0.0 || !finite(vv) || !finite(ev)) {
                breakdown();
                return;
            }
            if (f64)
                v.c3 = ev / vv;
            else
                v.c3_32 = (float)ev / (float)vv;
        }))
        return kLost;
    if (v.next != kGo) return (Step)v.next;
    const T c3 = f64 ? (T)v.c3 : (T)v.c3_32;
    if (threadIdx.x == kNT - 1) v.inv_rho = f64 ? 1.0 / (v.c2 * v.c3) : 0.0;
    typename Dot<T>::type d3[2] = {Dot<T>::zero(), Dot<T>::zero()};
    RES_ROWS(g, S.nb)
#pragma unroll
    for (int i = 0; i < BS; ++i) {
        const int o = S.own(sl, i);
        xs[o] = xs[o] + alpha * phs[o] + c3 * ehs[o];
        const T r = fma(-c3, S.collected(sl, i), rs[o]);
        rs[o] = r;
        Dot<T>::add(d3[0], r, r);
        Dot<T>::add(d3[1], r0s[o], r);
    }
    if (!g.template sum<2, false>(d3, [] {}, [&](double(&t)[2]) {
            const double rr = f64 ? t[0] : (double)(float)t[0], c1 = f64 ? t[1] : (double)(float)t[1];
            v.iter += 1;
            v.parity ^= 1;
            v.next = kGo;
            if (!finite(rr) || !finite(c1)) {
                if (f64) {
                    v.status = PFG_E_NONFINITE;
                    v.next = kDone;
                } else {
                    v.poisoned = 1;
                    breakdown();
                }
                return;
            }
            v.rr = rr;
            if (f64) {
                if (v.iter == 1) {
                    v.rr1 = rr;
                    v.goal1 = a.tol * a.tol * rr;
                    if (a.stop_rule == PFG_STOP_REFERENCE) v.exact |= !square_holds(a.tol, v.goal1);
                }
                if (a.stop_rule == PFG_STOP_REFERENCE ? reached<true>(v, a, rr) : reached<false>(v, a, rr))
                    v.next = kDone;
            } else if (replace_due(v, a, rr)) {
                v.next = kReplace;
            }
            if (v.next == kGo) {
                if (f64) {
                    if (v.c2 * v.c3 == 0.0) {
                        breakdown();
                    } else {
                        v.beta = quotient(c1, v.c2 * v.c3, v.inv_rho);
                        v.rho = c1;
                    }
                } else {
                    const float c2c3 = (float)v.c2 * v.c3_32;
                    if (c2c3 == 0.f) {
                        breakdown();
                    } else {
                        v.beta32 = (float)c1 / c2c3;
                        v.rho = c1;
                        v.breakdowns = 0;
                    }
                }
            }
            if (v.iter >= a.itrmax && v.next != kDone) {
                v.status = PFG_W_NOT_CONVERGED;
                v.next = kDone;
            }
        }))
        return kLost;
    return (Step)v.next;
}

template <typename T>
__device__ __forceinline__ T *take(unsigned char *&p, size_t n)
{
    T *q = reinterpret_cast<T *>(p);
    p += n * sizeof(T);
    return q;
}

// own vector <-> global rows
template <int BS, typename T>
__device__ void load_own(const Grid &g, int64_t nb, const T *v, T *o)
{
    RES_ROWS(g, nb)
#pragma unroll
    for (int i = 0; i < BS; ++i) o[(sl * BS + i) * 32 + g.lane] = v[(int64_t)BS * row + i];
}
template <int BS, typename T>
__device__ void store_own(const Grid &g, int64_t nb, T *v, const T *o)
{
    RES_ROWS(g, nb)
#pragma unroll
    for (int i = 0; i < BS; ++i) v[(int64_t)BS * row + i] = o[(sl * BS + i) * 32 + g.lane];
}
template <int BS, typename T>
__device__ void zero_own(const Grid &g, T *o)
{
    for (int sl = g.wid; sl < g.nsl; sl += kNW)
#pragma unroll
        for (int i = 0; i < BS; ++i) o[(sl * BS + i) * 32 + g.lane] = T(0);
}

// A CTA's own vectors: the first `a.near` of them (in the order of use per
// iteration) in shared memory, the others, and every one between two launches,
// in the scratch `home`, which has the same layout for the whole grid.
template <int BS, typename T>
struct Own {
    T *home;
    unsigned char *near;
    size_t n, all;
    int count;
    __device__ void init(const Grid &g, const ResArgs &a, int64_t ns, unsigned char *mem)
    {
        all = (size_t)ns * BS * 32;
        home = reinterpret_cast<T *>(a.home) + (size_t)g.s0 * BS * 32;
        n = (size_t)g.nsl * BS * 32;
        near = mem;
        count = a.near;
    }
    __device__ T *at(int k) const { return k < count ? reinterpret_cast<T *>(near) + k * n : home + k * all; }
    __device__ void copy(const Grid &g, int vectors, bool out) const
    {
        for (int k = 0; k < min(vectors, count); ++k) {
            T *s = reinterpret_cast<T *>(near) + k * n, *h = home + k * all;
            for (int sl = g.wid; sl < g.nsl; sl += kNW)
#pragma unroll
                for (int i = 0; i < BS; ++i) {
                    const int o = (sl * BS + i) * 32 + g.lane;
                    if (out)
                        h[o] = s[o];
                    else
                        s[o] = h[o];
                }
        }
    }
    // the rows' inverse diagonal blocks (planes: BS * BS of 32 per slice), in shared
    // memory as vectors k .. k + BS - 1 if those are
    __device__ const T *planes(const Grid &g, int k, const T *dinv, int64_t nb) const
    {
        const T *far = dinv + (size_t)g.s0 * (BS * BS * 32);
        if (k + BS > count) return far;
        T *o = reinterpret_cast<T *>(near) + k * n;
        RES_ROWS(g, nb)
#pragma unroll
        for (int e = 0; e < BS * BS; ++e)
            o[(sl * BS * BS + e) * 32 + g.lane] = __ldg(far + (sl * BS * BS + e) * 32 + g.lane);
        return o;
    }
};

// The CTA's share of the grid: slice pointers and segment table in shared memory.
struct Share {
    Grid g;
    Cut cut;
    unsigned char *wlo, *whi;
};

__device__ void open_share(Share &h, ResShared &sh, const ResArgs &a, const int64_t *sptr, unsigned char *&mem)
{
    Grid &g = h.g;
    g.sh = &sh;
    g.slots = a.slots;
    g.err = &a.st->err;
    g.lane = threadIdx.x & 31;
    g.wid = threadIdx.x >> 5;
    g.round = a.round;
    g.s0 = a.bounds[blockIdx.x];
    g.nsl = a.bounds[blockIdx.x + 1] - g.s0;
    int64_t *sp = take<int64_t>(mem, (size_t)g.nsl + 1 + ((g.nsl + 1) & 1));
    const size_t tab = ((size_t)g.nsl + 15) / 16 * 16;
    h.wlo = take<unsigned char>(mem, tab);
    h.whi = take<unsigned char>(mem, tab);
    for (int i = threadIdx.x; i <= g.nsl; i += kNT) sp[i] = sptr[g.s0 + i];
    if (threadIdx.x == 0) {
        sh.fail = 0;
        sh.state = *a.st;
    }
    h.cut.sp = sp;
    h.cut.nsl = g.nsl;
    __syncthreads();
    for (int sl = threadIdx.x; sl < g.nsl; sl += kNT) {
        const int t0 = (int)(sp[sl] - sp[0]), t1 = (int)(sp[sl + 1] - sp[0]);
        // (an empty slice takes the index between its neighbours' segments)
        const int n = h.cut.slots();
        h.wlo[sl] = n > 0 ? (unsigned char)h.cut.warp_of(min(t0, n - 1)) : 0;
        h.whi[sl] = t1 > t0 ? (unsigned char)h.cut.warp_of(t1 - 1) : kNoSegment;
    }
    __syncthreads();
}

template <int BS, typename T>
__device__ void open_solve(Solve<BS, T> &S, Share &h, T *buf, int64_t nb)
{
    S.g = &h.g;
    S.wlo = h.wlo;
    S.whi = h.whi;
    S.nb = nb;
    S.dinv = nullptr;
    S.buf = buf;
}

// ResState <-> Live, by one thread
__device__ void set_live(ResShared &sh, const ResArgs &a, bool by_reference)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        const ResState &s = sh.state;
        Live &v = sh.live;
        v.beta = s.beta;
        v.rho = s.rho;
        v.c2 = s.c2;
        v.c3 = s.c3;
        v.rr = s.rr;
        v.bb = s.bb;
        v.goal = a.tol < 0.0 ? -1.0 : a.tol * a.tol * s.bb;
        v.rr1 = s.rr1;
        v.goal1 = a.tol * a.tol * s.rr1;
        v.near0 = a.er0 * a.er0;
        v.exact = by_reference ? !square_holds(a.er0, v.near0) || (s.iter > 0 && !square_holds(a.tol, v.goal1))
                               : !square_holds(a.tol, v.goal);
        v.beta32 = (float)s.beta;
        v.c3_32 = (float)s.c3;
        v.rmax = s.rmax32;
        v.rmin = s.rmin32;
        v.iter = s.iter;
        v.parity = s.parity;
        v.status = s.status;
        v.breakdowns = s.breakdowns;
        v.poisoned = s.poisoned;
    }
    __syncthreads();
}
template <typename T>
__device__ void keep_live(ResShared &sh)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        ResState &s = sh.state;
        const Live &v = sh.live;
        s.beta = sizeof(T) == 8 ? v.beta : (double)v.beta32;
        s.rho = v.rho;
        s.c2 = v.c2;
        s.c3 = sizeof(T) == 8 ? v.c3 : (double)v.c3_32;
        s.rr = v.rr;
        s.rr1 = v.rr1;
        s.rmax32 = v.rmax;
        s.rmin32 = v.rmin;
        s.iter = v.iter;
        s.parity = v.parity;
        s.status = v.status;
        s.breakdowns = v.breakdowns;
        s.poisoned = v.poisoned;
    }
    __syncthreads();
}
// every thread holds the same s
__device__ void put_state(ResShared &sh, const ResState &s)
{
    __syncthreads();
    if (threadIdx.x == 0) sh.state = s;
    __syncthreads();
}
__device__ void close_state(ResShared &sh, const Grid &g, const ResArgs &a, int phase)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sh.state.phase = phase;
        sh.state.round = g.round;
        sh.state.err = *(volatile int *)&a.st->err;
        *a.st = sh.state;
    }
}

// out(sl, i, b - A x) for the CTA's rows, s.true_rr, s.bb and s.rel.  x is
// published by the call.
template <int BS, typename Prod, typename Out>
__device__ bool true_residual(const Solve<BS, double> &S, const ResArgs &a, ResState &s, const Prod &product,
                              const Out &out)
{
    Grid &g = *S.g;
    if (!g.barrier()) return false;
    product([&](int c, double(&v)[BS]) {
#pragma unroll
        for (int i = 0; i < BS; ++i) v[i] = a.x[(int64_t)BS * c + i];
    });
    double d[2] = {0.0, 0.0};
    RES_ROWS(g, S.nb)
    {
        double q[BS];
        S.collect(sl, q);
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            const double b = __ldg(a.b + (int64_t)BS * row + i);
            const double r = b - q[i];
            out(sl, i, r);
            d[0] = fma(r, r, d[0]);
            d[1] = fma(b, b, d[1]);
        }
    }
    if (!g.template sum<2, false>(d, [] {}, [](double(&)[2]) {})) return false;
    s.true_rr = d[0];
    s.bb = d[1];
    s.rel = d[1] > 0.0 ? sqrt(d[0]) / sqrt(d[1]) : sqrt(d[0]);
    return true;
}

// FP64 solve: run_cg64 / run_bicgstab64 of krylov.cu, restarts from the true
// residual included.
template <int BS, bool CG>
__device__ void solve64(Solve<BS, double> &S, ResShared &sh, const ResArgs &a, unsigned char *mem)
{
    Grid &g = *S.g;
    const int64_t nb = S.nb;
    Own<BS, double> own;
    own.init(g, a, a.A64.ns, mem);
    const bool pc = a.pc != PFG_PC_NONE;
    // CG: r, p, x; BiCGSTAB: r, y, p, r0, x, M^-1 p, M^-1 e (unpreconditioned: p and
    // e themselves; e shares r's place until r is formed from it, so x is advanced
    // before r is written); then the inverse diagonal blocks
    double *rs = own.at(0), *ps = own.at(CG ? 1 : 2), *xs = own.at(CG ? 2 : 4);
    double *ys = CG ? nullptr : own.at(1), *r0s = CG ? nullptr : own.at(3);
    double *phs = !CG && pc ? own.at(5) : ps, *ehs = !CG && pc ? own.at(6) : rs;
    const int vectors = CG ? 3 : (pc ? 7 : 5);
    if (pc) S.dinv = own.planes(g, vectors, a.dinv64, nb);
    bool resumed = sh.state.phase == 1;
    if (resumed)
        own.copy(g, vectors, false);
    else
        load_own<BS>(g, nb, a.x, xs);
    const int max_restarts = !CG && a.stop_rule == PFG_STOP_REFERENCE ? 1 : 20;
    int left = a.budget;
    for (;;) {
        if (!resumed) {
            ResState s = sh.state;
            store_own<BS>(g, nb, a.x, xs);
            if (!true_residual<BS>(
                    S, a, s, [&](const auto &src) { S.product(src); },
                    [&](int sl, int i, double r) { rs[S.own(sl, i)] = r; }))
                return;
            const bool stop = (CG || a.stop_rule == PFG_STOP_TRUE_RELATIVE) && s.rel <= a.tol;
            if (stop || s.status != PFG_OK || s.restart >= max_restarts) {
                put_state(sh, s);
                break;
            }
            s.restart += 1;
            zero_own<BS>(g, ps);
            if (!CG) zero_own<BS>(g, ys);
            double d[2] = {0.0, 0.0};
            RES_ROWS(g, nb)
            {
                double r[BS], z[BS];
#pragma unroll
                for (int i = 0; i < BS; ++i) r[i] = rs[S.own(sl, i)];
                if (CG) {
                    S.precond(sl, r, z);
                    publish<BS>(a.pub64[0], row, z);
#pragma unroll
                    for (int i = 0; i < BS; ++i) ps[S.own(sl, i)] = z[i];
                } else {
#pragma unroll
                    for (int i = 0; i < BS; ++i) {
                        r0s[S.own(sl, i)] = r[i];
                        z[i] = r[i];
                    }
                }
#pragma unroll
                for (int i = 0; i < BS; ++i) {
                    d[0] = fma(r[i], z[i], d[0]);
                    d[1] = fma(r[i], r[i], d[1]);
                }
            }
            if (!g.template sum<2, true>(d, [] {}, [](double(&)[2]) {})) return;
            s.rho = d[0];
            s.rr = d[1];
            s.beta = 0.0;
            s.c3 = 0.0;
            put_state(sh, s);
        }
        resumed = false;
        set_live(sh, a, !CG && a.stop_rule == PFG_STOP_REFERENCE);
        Step st = kGo;
        while (st == kGo && left > 0) {
            st = CG ? cg_step(S, a, xs, rs, ps, (double *)nullptr, a.pub64[0], (double *)nullptr, (double *)nullptr,
                              (double *)nullptr)
                    : bicg_step(S, a, xs, rs, r0s, ps, ys, phs, ehs, a.pub64[0], a.pub64[1]);
            --left;
        }
        if (st == kLost) return;
        keep_live<double>(sh);
        if (st == kGo) {  // out of budget: the next launch goes on
            own.copy(g, vectors, true);
            close_state(sh, g, a, 1);
            return;
        }
    }
    close_state(sh, g, a, 2);
}

template <int BS, bool CG>
__global__ void __launch_bounds__(kNT, 1) k_resident64(const ResArgs a)
{
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ ResShared sh;
    __shared__ __align__(8) uint64_t bars[kNW * kMaxStages];
    unsigned char *mem = dsm;
    unsigned char *ring = take<unsigned char>(mem, (size_t)kNW * a.stages * kStageBytes<BS, double>);
    Share h;
    open_share(h, sh, a, a.A64.sptr, mem);
    Solve<BS, double> S;
    open_solve(S, h, take<double>(mem, (size_t)(h.g.nsl + kNW) * BS * 32), a.A64.nb);
    S.mat.init(a.A64, h.cut, bars, ring, a.stages);
    solve64<BS, CG>(S, sh, a, mem);
    S.mat.drain();
}

// Mixed solve: run_mixed of krylov.cu (FP32 iterations, the residual replaced by
// the FP64 one, corrections kept only if they lower it, hand-over to FP64).
template <int BS, bool CG>
__device__ void solve_mixed(Solve<BS, float> &S, Solve<BS, double> &D, const Cut &cut, ResShared &sh,
                            const ResArgs &a, unsigned char *mem)
{
    Grid &g = *S.g;
    const int64_t nb = S.nb;
    Own<BS, float> own;
    own.init(g, a, a.A32.ns, mem);
    const bool pc = a.pc != PFG_PC_NONE;
    // CG: r, z, p, x; BiCGSTAB as in solve64
    float *rs = own.at(0), *ps = own.at(2), *xs = own.at(CG ? 3 : 4);
    float *zs = CG ? own.at(1) : nullptr, *ys = CG ? nullptr : own.at(1), *r0s = CG ? nullptr : own.at(3);
    float *phs = !CG && pc ? own.at(5) : ps, *ehs = !CG && pc ? own.at(6) : rs;
    const int vectors = CG ? 4 : (pc ? 7 : 5);
    if (pc) S.dinv = own.planes(g, vectors, a.dinv32, nb);
    bool resumed = sh.state.phase == 1;
    if (resumed) {
        own.copy(g, vectors, false);
    } else {
        zero_own<BS>(g, xs);
        zero_own<BS>(g, ps);
        if (!CG) zero_own<BS>(g, ys);
    }
    // r32 = the FP64 residual
    auto residual = [&](ResState &s) {
        return true_residual<BS>(
            D, a, s,
            [&](const auto &src) {
                apply_plain<BS>(a.A64, cut, src, D.buf);
                __syncthreads();
            },
            [&](int sl, int i, double r) { rs[S.own(sl, i)] = (float)r; });
    };
    // x += x32 (x kept in xb when `backup`), x32 = 0
    auto fold = [&](bool backup) {
        RES_ROWS(g, nb)
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            const int64_t j = (int64_t)BS * row + i;
            const double x = a.x[j];
            if (backup) a.xb[j] = x;
            a.x[j] = x + (double)xs[S.own(sl, i)];
            xs[S.own(sl, i)] = 0.f;
        }
    };
    int left = a.budget;
    for (;;) {
        if (!resumed) {
            ResState s = sh.state;
            bool rejected = false;
            if (!s.first) {
                if (s.poisoned) {  // an overflowed correction is dropped
                    zero_own<BS>(g, xs);
                    s.poisoned = 0;
                    rejected = true;
                } else {
                    fold(true);
                }
            }
            if (!residual(s)) return;
            const double growth = CG ? 1.0 : 10.0;
            if (!s.first && !rejected && !(s.rel < growth * s.prev_rel)) {
                RES_ROWS(g, nb)
#pragma unroll
                for (int i = 0; i < BS; ++i) a.x[(int64_t)BS * row + i] = a.xb[(int64_t)BS * row + i];
                if (!residual(s)) return;
                rejected = true;
            }
            s.prev_rel = s.rel;
            s.failures = rejected ? s.failures + 1 : 0;
            if (rejected && s.rel < 100.0 * a.tol && CG) s.failures = max(s.failures, kReject);
            bool give_up = s.failures >= kReject && s.rel > a.tol;
            if (!give_up) {
                if (s.first || s.rel < 0.9 * s.best_rel) {
                    s.best_rel = s.rel;
                    s.stall = 0;
                } else if (++s.stall >= (CG ? kStallCG : kStallBiCG) && s.rel > a.tol) {
                    give_up = true;
                }
            }
            if (give_up) {
                s.fallback = 1;
                put_state(sh, s);
                break;
            }
            s.replacements += 1;
            const bool conv = sqrt(s.true_rr) <= a.tol * sqrt(s.bb);
            if (CG) {
                const bool keep = !s.first && !rejected;
                if (rejected) zero_own<BS>(g, ps);
                if (!keep) {  // the gather reads the previous p even where beta is 0
                    float *pold = a.pub32[s.parity ? 2 : 1];
                    const float none[BS] = {};
                    RES_ROWS(g, nb) publish<BS>(pold, row, none);
                }
                Comp32 d[2] = {Comp32{0.f, 0.f}, Comp32{0.f, 0.f}};
                RES_ROWS(g, nb)
                {
                    float r[BS], z[BS];
#pragma unroll
                    for (int i = 0; i < BS; ++i) r[i] = rs[S.own(sl, i)];
                    S.precond(sl, r, z);
                    publish<BS>(a.pub32[0], row, z);
#pragma unroll
                    for (int i = 0; i < BS; ++i) {
                        zs[S.own(sl, i)] = z[i];
                        comp_add_prod(d[0], r[i], z[i]);
                        comp_add_prod(d[1], r[i], r[i]);
                    }
                }
                if (!g.template sum<2, true>(d, [] {}, [](double(&)[2]) {})) return;
                const float rho = (float)sh.tot[(g.round - 1) & 1][0];
                s.rr = (double)(float)sh.tot[(g.round - 1) & 1][1];
                s.beta = keep && s.rho != 0.0 ? (double)(rho / (float)s.rho) : 0.0;
                s.rho = (double)rho;
            } else {
                bool full = s.first || rejected || s.breakdowns > 0;
                for (;;) {
                    if (full) {
                        zero_own<BS>(g, ps);
                        zero_own<BS>(g, ys);
                    }
                    Comp32 d[2] = {Comp32{0.f, 0.f}, Comp32{0.f, 0.f}}, d0[1] = {Comp32{0.f, 0.f}};
                    RES_ROWS(g, nb)
#pragma unroll
                    for (int i = 0; i < BS; ++i) {
                        const int o = S.own(sl, i);
                        const float r = rs[o];
                        if (full) r0s[o] = r;
                        const float q = full ? r : r0s[o];
                        comp_add_prod(d[0], q, r);
                        comp_add_prod(d[1], r, r);
                        comp_add_prod(d0[0], q, q);
                    }
                    if (!g.template sum<2, true>(d, [] {}, [](double(&)[2]) {})) return;
                    const float c1 = (float)sh.tot[(g.round - 1) & 1][0], rr = (float)sh.tot[(g.round - 1) & 1][1];
                    if (!g.template sum<1, false>(d0, [] {}, [](double(&)[1]) {})) return;
                    const float r0r0 = (float)sh.tot[(g.round - 1) & 1][0];
                    const float c2c3 = (float)s.c2 * (float)s.c3;
                    s.beta = !full && c2c3 != 0.f ? (double)(c1 / c2c3) : 0.0;
                    if (full) s.c3 = 0.0;
                    s.rho = (double)c1;
                    s.rr = (double)rr;
                    if (full) break;
                    // keep direction and shadow residual while r0.r carries FP32 digits
                    const double den = sqrt((double)rr * (double)r0r0);
                    full = !(den > 0.0 && fabs((double)c1) > 1e-3 * den);
                    if (!full) break;
                }
            }
            s.rmax32 = s.rmin32 = sqrtf((float)s.rr);
            s.first = 0;
            if (s.breakdowns > 3 && !conv) s.fallback = 1;
            put_state(sh, s);
            if (conv || s.fallback) break;
        }
        resumed = false;
        set_live(sh, a, false);
        Step st = kGo;
        while (st == kGo && left > 0) {
            st = CG ? cg_step(S, a, xs, rs, ps, zs, (float *)nullptr, a.pub32[0], a.pub32[1], a.pub32[2])
                    : bicg_step(S, a, xs, rs, r0s, ps, ys, phs, ehs, a.pub32[0], a.pub32[1]);
            --left;
        }
        if (st == kLost) return;
        keep_live<float>(sh);
        if (st == kGo) {
            own.copy(g, vectors, true);
            close_state(sh, g, a, 1);
            return;
        }
        if (st == kDone) {  // breakdown or itrmax: fold what was computed
            fold(false);
            ResState s = sh.state;
            if (!residual(s)) return;
            put_state(sh, s);
            break;
        }
    }
    close_state(sh, g, a, 2);
}

template <int BS, bool CG>
__global__ void __launch_bounds__(kNT, 1) k_resident_mixed(const ResArgs a)
{
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ ResShared sh;
    __shared__ __align__(8) uint64_t bars[kNW * kMaxStages];
    unsigned char *mem = dsm;
    unsigned char *ring = take<unsigned char>(mem, (size_t)kNW * a.stages * kStageBytes<BS, float>);
    Share h;
    open_share(h, sh, a, a.A32.sptr, mem);
    // both products' segment sums (never at once)
    double *buf = take<double>(mem, (size_t)(h.g.nsl + kNW) * BS * 32);
    Solve<BS, double> D;
    Solve<BS, float> S;
    open_solve(D, h, buf, a.A64.nb);
    open_solve(S, h, reinterpret_cast<float *>(buf), a.A32.nb);
    S.mat.init(a.A32, h.cut, bars, ring, a.stages);
    solve_mixed<BS, CG>(S, D, h.cut, sh, a, mem);
    S.mat.drain();
}

using ResKernel = void (*)(ResArgs);

ResKernel pick_kernel(int bs, int algorithm, bool mixed)
{
    const bool cg = algorithm == PFG_ALG_CG;
    if (mixed)
        return bs == 3 ? (cg ? k_resident_mixed<3, true> : k_resident_mixed<3, false>)
                       : (cg ? k_resident_mixed<1, true> : k_resident_mixed<1, false>);
    return bs == 3 ? (cg ? k_resident64<3, true> : k_resident64<3, false>)
                   : (cg ? k_resident64<1, true> : k_resident64<1, false>);
}

}  // namespace

// Work of a slice: its slots, and about four slots' worth of row updates.
constexpr int64_t kRowWork = 4;

void share_slices(DevMatrix &A, int ctas, cudaStream_t st)
{
    if (A.ns <= 0) return;
    const int64_t G = std::min<int64_t>(A.ns, std::min(ctas > 0 ? ctas : sm_count_device(), kResMaxCtas));
    if (A.share_ctas == G) return;
    A.share_ctas = 0;
    std::vector<int64_t> sp((size_t)A.ns + 1);
    PFG_CUDA(cudaMemcpyAsync(sp.data(), A.sptr.p, sp.size() * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    PFG_CUDA(cudaStreamSynchronize(st));
    const double total = (double)(sp[(size_t)A.ns] + kRowWork * A.ns);
    std::vector<int> b((size_t)G + 1, 0);
    int64_t s = 0, most = 0;
    for (int64_t c = 1; c <= G; ++c) {
        const double goal = total * (double)c / (double)G;
        const int64_t first = s;
        // to the slice boundary nearest the goal, at least one slice for this CTA and each later one
        while (s < A.ns - (G - c) && (s == first || (double)(sp[(size_t)s + 1] + sp[(size_t)s]) / 2.0 +
                                                            (double)kRowWork * ((double)s + 0.5) <= goal))
            ++s;
        if (c == G) s = A.ns;
        b[(size_t)c] = (int)s;
        most = std::max(most, s - first);
    }
    A.share.resize((size_t)G + 1);
    PFG_CUDA(cudaMemcpyAsync(A.share.p, b.data(), b.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    PFG_CUDA(cudaStreamSynchronize(st));
    A.share_ctas = (int)G;
    A.share_max = (int)most;
}

ResPlan plan_resident(const DevMatrix &A, int algorithm, bool mixed, bool precond)
{
    ResPlan pl;
    if (A.share_ctas <= 0) return pl;
    const bool cg = algorithm == PFG_ALG_CG;
    const size_t per = (size_t)A.share_max, plane = (size_t)A.bs * 32, word = mixed ? 4 : 8;
    pl.vectors = (cg ? (mixed ? 4 : 3) : (precond ? 7 : 5)) + (precond ? A.bs : 0);
    const size_t fixed = (per + 2) * 8 + 2 * (per + 15) + (per + kNW) * plane * 8 + 64;
    const size_t vec = per * plane * word;
    const size_t stage = (size_t)kNW * (mixed ? (A.bs == 3 ? kStageBytes<3, float> : kStageBytes<1, float>)
                                              : (A.bs == 3 ? kStageBytes<3, double> : kStageBytes<1, double>));
    if (fixed + 2 * stage > kSmemMax) return pl;
    // a few stages first (a copy takes about as long as two chunks), then the
    // vectors in the order of their use, then stages again with what is left
    int stages = 2;
    while (stages < (mixed ? 2 : 4) && fixed + (size_t)(stages + 1) * stage <= kSmemMax) ++stages;
    int near = (int)std::min<size_t>((kSmemMax - fixed - (size_t)stages * stage) / std::max<size_t>(vec, 1),
                                     (size_t)pl.vectors);
    while (stages < kMaxStages && fixed + (size_t)near * vec + (size_t)(stages + 1) * stage <= kSmemMax) ++stages;
    pl.ctas = A.share_ctas;
    pl.stages = stages;
    pl.near = near;
    pl.smem = fixed + (size_t)near * vec + (size_t)stages * stage;
    pl.home_bytes = (size_t)(pl.vectors - (precond ? A.bs : 0)) * (size_t)A.ns * plane * word;
    return pl;
}

std::shared_ptr<ResDevice> ResDevice::current()
{
    static std::mutex mu;
    static std::weak_ptr<ResDevice> known[64];
    int dev = 0;
    PFG_CUDA(cudaGetDevice(&dev));
    PFG_CHECK(dev >= 0 && dev < 64, PFG_E_UNSUPPORTED, "device ordinal above 63");
    std::lock_guard<std::mutex> lk(mu);
    std::shared_ptr<ResDevice> d = known[dev].lock();
    if (!d) {
        d = std::make_shared<ResDevice>();
        d->slots.alloc(kResSlots);
        PFG_CUDA(cudaEventCreateWithFlags(&d->last, cudaEventDisableTiming));
        known[dev] = d;
    }
    return d;
}

namespace {

// The launch, after the one before on this device.  Its inboxes are those that a launch
// of as many CTAs left, each buffer in the state that the next round expects, or empty
// ones (a memset of at most 3 MB) where another grid was there last or may still be.
// Its number; 0: the device does not hold the grid at once.
uint64_t launch_in_turn(ResDevice &dev, ResKernel kern, int ctas, ResArgs &a, size_t smem, cudaStream_t st)
{
    std::lock_guard<std::mutex> lk(dev.mu);
    const bool ready = dev.in_flight == 0 && dev.ready_ctas == ctas;
    dev.ready_ctas = 0;
    if (ready) {
        a.round = dev.ready_round;
    } else {
        if (dev.in_flight > 0) PFG_CUDA(cudaStreamWaitEvent(st, dev.last, 0));
        constexpr size_t inbox = (size_t)kResValues * kResMaxCtas * sizeof(double);
        PFG_CUDA(cudaMemset2DAsync(dev.slots.p, kResMaxCtas * inbox, 0xff, ctas * inbox, kResRounds, st));
        a.round = 0;
    }
    void *args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)kern, dim3(ctas), dim3(kNT), args, smem, st);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        (void)cudaGetLastError();
        return 0;
    }
    PFG_CUDA(e);
    ++dev.in_flight;
    ++dev.launches;
    PFG_CUDA(cudaEventRecord(dev.last, st));
    return dev.launches;
}

// Waits for launch `number`; its state in *host.
void end_turn(ResDevice &dev, uint64_t number, int ctas, const ResState *host, cudaStream_t st)
{
    const cudaError_t e = cudaStreamSynchronize(st);
    std::lock_guard<std::mutex> lk(dev.mu);
    --dev.in_flight;
    if (number == dev.launches && e == cudaSuccess && host->err == 0) {
        dev.ready_ctas = ctas;
        dev.ready_round = host->round;
    }
    PFG_CUDA(e);
}

}  // namespace

int run_resident_kernel(ResDevice &dev, const ResPlan &pl, ResArgs a, int bs, int algorithm, bool mixed,
                        ResState *host, bool debug, cudaStream_t st)
{
    const ResKernel kern = pick_kernel(bs, algorithm, mixed);
    PFG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
    a.stages = pl.stages;
    a.near = pl.near;
    a.slots = dev.slots.p;
    PFG_CUDA(cudaMemcpyAsync(a.st, host, sizeof(ResState), cudaMemcpyHostToDevice, st));
    for (int launches = 1;; ++launches) {
        const uint64_t number = launch_in_turn(dev, kern, pl.ctas, a, pl.smem, st);
        if (number == 0) {
            PFG_CHECK(launches == 1, PFG_E_CUDA, "resident solve: the device took no further launch");
            return 0;
        }
        const cudaError_t e = cudaMemcpyAsync(host, a.st, sizeof(ResState), cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) host->err = 1;
        end_turn(dev, number, pl.ctas, host, st);
        PFG_CUDA(e);
        PFG_CHECK(host->err == 0, PFG_E_INTERNAL, "resident solve: a wait between CTAs ran out");
        if (debug && mixed)
            fprintf(stderr, "[pfg] mixed iter %d replacement %d |b-Ax|/|b| %.3e%s\n", host->iter, host->replacements,
                    host->rel, host->fallback ? ", hand-over to FP64" : "");
        else if (debug)
            fprintf(stderr, "[pfg] %s iter %d |r| %.3e\n", algorithm == PFG_ALG_CG ? "CG64" : "BiCGSTAB64", host->iter,
                    sqrt(host->rr));
        if (host->phase == 2) return launches;
    }
}

}  // namespace pfg
