// sell.cu -- block-row (BCRS) -> sliced-ELL conversion on the device.
#include "assembly.cuh"

namespace pfg {

// width of each slice = longest block row in it
__global__ void k_sell_widths(int64_t nb, int64_t ns, const int64_t *__restrict__ rp, int64_t *__restrict__ width)
{
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += (int64_t)gridDim.x * blockDim.x) {
        int64_t w = 0;
        for (int l = 0; l < 32; ++l) {
            const int64_t row = s * 32 + l;
            if (row < nb) w = max(w, rp[row + 1] - rp[row]);
        }
        width[s] = w;
    }
}

// one thread per (slice, lane): block columns, padding points at the row itself
__global__ void k_sell_pattern(int64_t nb, int64_t ns, const int64_t *__restrict__ rp, const int *__restrict__ bcol,
                               const int64_t *__restrict__ sptr, int *__restrict__ scol)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ns * 32; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = t >> 5;
        const int l = (int)(t & 31);
        const int64_t row = t;
        const int64_t b0 = sptr[s], w = sptr[s + 1] - b0;
        const int64_t r0 = row < nb ? rp[row] : 0;
        const int64_t nblk = row < nb ? rp[row + 1] - r0 : 0;
        const int self = row < nb ? (int)row : 0;
        for (int64_t k = 0; k < w; ++k) scol[(b0 + k) * 32 + l] = k < nblk ? bcol[r0 + k] : self;
    }
}

// Slice values: a warp per (slice, entry plane), so a 3x3-block slice is a CTA of
// nine warps; kTileK slots at a time through a shared-memory tile of the warp.  Each
// row's plane is read as one contiguous run of its blocks (block row layout,
// bsr.cuh), eight rows' loads in flight, and written back slot by slot as 32
// consecutive lanes; FP64 and FP32 copies come from one read.  Bound by HBM on
// large meshes, by the latency of the 32 row reads on small ones: a warp per slice
// that took the nine planes in turn ran 831 us at 274,625 rows (FP64 copy) and 157 us
// at 4,032; this runs 230 us and 12 us (1.1 GB moved: 4.9 TB/s).
constexpr int kTileK = 32;

template <int BS>
constexpr int kSellSlices = BS == 3 ? 1 : 8;  // slices per CTA
template <int BS>
constexpr int kSellThreads = 32 * BS * BS * kSellSlices<BS>;
template <int BS>
constexpr size_t kSellTile = (size_t)BS * BS * kSellSlices<BS> * 32 * (kTileK + 1) * sizeof(double);

template <int BS>
__global__ void __launch_bounds__(kSellThreads<BS>)
    k_sell_values(int64_t nb, int64_t ns, const int64_t *__restrict__ rp, const double *__restrict__ v64,
                  const int64_t *__restrict__ sptr, double *__restrict__ s64, float *__restrict__ s32)
{
    constexpr int BB = BS * BS;
    extern __shared__ double dyn_tile[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double *tile = dyn_tile + (size_t)w * 32 * (kTileK + 1);
    const int e = w % BB;
    for (int64_t s = (int64_t)blockIdx.x * kSellSlices<BS> + w / BB; s < ns; s += (int64_t)gridDim.x * kSellSlices<BS>) {
        const int64_t b0 = sptr[s];
        const int wdt = (int)(sptr[s + 1] - b0);
        const int64_t row = s * 32 + lane;
        const int64_t r0 = row < nb ? rp[row] : 0;
        const int nblk = row < nb ? (int)(rp[row + 1] - r0) : 0;
        for (int kc = 0; kc < wdt; kc += kTileK) {
#pragma unroll 8
            for (int l = 0; l < 32; ++l) {
                const int64_t r0l = __shfl_sync(0xffffffffu, r0, l);
                const int nl = __shfl_sync(0xffffffffu, nblk, l);
                const int k = kc + lane;
                tile[l * (kTileK + 1) + lane] = k < nl ? ld_stream(v64 + r0l * BB + (int64_t)e * nl + k) : 0.0;
            }
            __syncwarp();
            const int kend = min(kTileK, wdt - kc);
#pragma unroll 4
            for (int kk = 0; kk < kend; ++kk) {
                const double v = tile[lane * (kTileK + 1) + kk];
                const int64_t o = ((b0 + kc + kk) * BB + e) * 32 + lane;
                if (s64) s64[o] = v;
                if (s32) s32[o] = (float)v;
            }
            __syncwarp();
        }
    }
}

template <int BS>
static void launch_sell_values(DevMatrix &A, double *s64, float *s32, cudaStream_t st)
{
    PFG_CUDA(cudaFuncSetAttribute(k_sell_values<BS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSellTile<BS>));
    const int64_t ctas = (A.ns + kSellSlices<BS> - 1) / kSellSlices<BS>;
    k_sell_values<BS><<<(int)std::min<int64_t>(ctas, sm_count_device() * 16), kSellThreads<BS>, kSellTile<BS>, st>>>(
        A.nb, A.ns, A.rp.p, A.v64.p, A.sptr.p, s64, s32);
    PFG_CUDA(cudaGetLastError());
}

void build_sell(DevMatrix &A, bool want64, bool want32, cudaStream_t st)
{
    PFG_CHECK(A.nb > 0, PFG_E_STATE, "empty matrix");
    const int g = grid_for(A.nb, 256, sm_count_device() * 16);
    if (!A.sell_pattern) {
        A.ns = (A.nb + 31) / 32;
        DevBuf<int64_t> width((size_t)A.ns + 1);
        PFG_CUDA(cudaMemsetAsync(width.p, 0, (A.ns + 1) * sizeof(int64_t), st));
        k_sell_widths<<<grid_for(A.ns, 256, sm_count_device() * 16), 256, 0, st>>>(A.nb, A.ns, A.rp.p, width.p);
        PFG_CUDA(cudaGetLastError());
        A.sptr.resize((size_t)A.ns + 1);
        const int64_t slots = exclusive_scan(width.p, A.sptr.p, A.ns + 1, st);
        A.scol.resize((size_t)std::max<int64_t>(slots * 32, 1));
        k_sell_pattern<<<g, 256, 0, st>>>(A.nb, A.ns, A.rp.p, A.col.p, A.sptr.p, A.scol.p);
        PFG_CUDA(cudaGetLastError());
        A.sell_pattern = true;
        A.s64_valid = A.s32_valid = false;
    }
    const bool do64 = want64 && !A.s64_valid, do32 = want32 && !A.s32_valid;
    if (!do64 && !do32) return;  // up to date
    const size_t nv = A.scol.n * (size_t)(A.bs * A.bs);
    if (do64) A.s64.resize(nv);
    if (do32) A.s32.resize(nv);
    if (A.bs == 3)
        launch_sell_values<3>(A, do64 ? A.s64.p : nullptr, do32 ? A.s32.p : nullptr, st);
    else
        launch_sell_values<1>(A, do64 ? A.s64.p : nullptr, do32 ? A.s32.p : nullptr, st);
    A.s64_valid |= do64;
    A.s32_valid |= do32;
}

// ------------------------------------------------- upper half (symmetric storage)
// width of each slice = most upper blocks (column >= row) of a row in it
__global__ void k_sellu_widths(int64_t nb, int64_t ns, const int64_t *__restrict__ rp, const int *__restrict__ bcol,
                               int64_t *__restrict__ width)
{
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += (int64_t)gridDim.x * blockDim.x) {
        int64_t w = 0;
        for (int l = 0; l < 32; ++l) {
            const int64_t row = s * 32 + l;
            if (row >= nb) break;
            int64_t c = 0;
            for (int64_t k = rp[row]; k < rp[row + 1]; ++k) c += bcol[k] >= row;
            w = max(w, c);
        }
        width[s] = w;
    }
}

// Columns and FP32 values of the upper blocks (column >= row) of each row, in
// the row's order; padding slots point at the row itself with zero values.
// A CTA of nine warps per slice, kTileK slots at a time: the warps share out the
// rows to find, by the ballot prefix of "upper" over a row's blocks, which block
// fills each slot (kept in shared memory); then each warp copies one entry plane
// as k_sell_values does.  (One warp per slice: 811 us at 274,625 rows; this: 298 us.)
__global__ void __launch_bounds__(288)
    k_sellu_fill(int64_t nb, int64_t ns, const int64_t *__restrict__ rp, const int *__restrict__ bcol,
                 const double *__restrict__ v64, const int64_t *__restrict__ sptr, int *__restrict__ scol,
                 float *__restrict__ sval)
{
    __shared__ short kmap[32][kTileK];
    __shared__ int ucnt[32];
    __shared__ float tiles[9][32][kTileK + 1];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int64_t s = blockIdx.x; s < ns; s += gridDim.x) {
        const int64_t b0 = sptr[s];
        const int wdt = (int)(sptr[s + 1] - b0);
        const int64_t row = s * 32 + lane;
        const int64_t r0 = row < nb ? rp[row] : 0;
        const int nblk = row < nb ? (int)(rp[row + 1] - r0) : 0;
        for (int kc = 0; kc < wdt; kc += kTileK) {
            // slots [kc, kc + kTileK) of every row: which of its blocks fill them
#pragma unroll 4
            for (int l = w; l < 32; l += 9) {
                const int64_t r0l = __shfl_sync(0xffffffffu, r0, l);
                const int nl = __shfl_sync(0xffffffffu, nblk, l);
                const int64_t rowl = s * 32 + l;
                int base = 0;
                for (int k0 = 0; k0 < nl; k0 += 32) {
                    const int k = k0 + lane;
                    const bool up = k < nl && bcol[r0l + k] >= rowl;
                    const unsigned bal = __ballot_sync(0xffffffffu, up);
                    const int pos = base + __popc(bal & ((1u << lane) - 1u)) - kc;
                    if (up && pos >= 0 && pos < kTileK) kmap[l][pos] = (short)k;
                    base += __popc(bal);
                }
                if (lane == 0) ucnt[l] = min(max(base - kc, 0), kTileK);
            }
            __syncthreads();
            const int kend = min(kTileK, wdt - kc);
            const int mine = ucnt[lane];
            for (int kk = w; kk < kend; kk += 9)
                scol[(b0 + kc + kk) * 32 + lane] = kk < mine ? bcol[r0 + kmap[lane][kk]] : (row < nb ? (int)row : 0);
            float(*tile)[kTileK + 1] = tiles[w];
#pragma unroll 8
            for (int l = 0; l < 32; ++l) {
                const int64_t r0l = __shfl_sync(0xffffffffu, r0, l);
                const int nl = __shfl_sync(0xffffffffu, nblk, l);
                tile[l][lane] = lane < ucnt[l] ? (float)v64[r0l * 9 + (int64_t)w * nl + kmap[l][lane]] : 0.f;
            }
            __syncwarp();
#pragma unroll 4
            for (int kk = 0; kk < kend; ++kk) sval[((b0 + kc + kk) * 9 + w) * 32 + lane] = tile[lane][kk];
            __syncthreads();  // kmap and ucnt are rewritten for the next slots
        }
    }
}

// Counts the upper blocks (i, j) whose transpose partner (j, i) is missing or
// differs by more than 1e-9 relative (plus 1e-12 of the diagonal scale of the
// two rows: assembly rounding leaves noise in entries that cancel to zero).
// One warp per row i, three of its upper blocks at a time: the warp reads row j's
// block columns (one load per 32) and votes for the slot of (j, i); then 27 lanes
// compare the three blocks' entries.  Finite entries with the same bits -- all of an
// assembled and eliminated matrix's -- need no arithmetic: nine FP64 comparisons
// for every block kept GB300's FP64 pipe busy for most of the 950 us this took at
// 274,625 rows (4,032 rows: 297 us); now 425 us and 11 us.
// A diagonal block is no pair and may be anything: *skew is raised where one is not
// symmetric itself, by the same measure.
__global__ void k_sym_check(int64_t nb, const int64_t *__restrict__ rp, const int *__restrict__ bcol,
                            const double *__restrict__ v64, unsigned long long *__restrict__ bad,
                            unsigned long long *__restrict__ skew)
{
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    // this lane's entry (r, c) of block `u` of three
    const int u3 = min(lane / 9, 2), e3 = lane - 9 * (lane / 9), r3 = e3 / 3, c3 = e3 - 3 * r3;
    // largest |entry| of a row's diagonal block (the warp's lanes share the search)
    auto diag_scale = [&](int64_t i) {
        const int64_t r0 = rp[i];
        const int n = (int)(rp[i + 1] - r0);
        double d = 0.0;
        for (int k = lane; k < n; k += 32)
            if (bcol[r0 + k] == i)
                for (int e = 0; e < 9; e += 4) d = fmax(d, fabs(v64[r0 * 9 + (int64_t)e * n + k]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d = fmax(d, __shfl_xor_sync(0xffffffffu, d, o));
        return d;
    };
    for (int64_t i = w0; i < nb; i += nw) {
        const int64_t ri = rp[i];
        const int ni = (int)(rp[i + 1] - ri);
        unsigned long long nbad = 0;
        for (int k0 = 0; k0 < ni; k0 += 32) {
            const int mine = k0 + lane < ni ? bcol[ri + k0 + lane] : -1;
            if (mine == i) {
                const double *v = v64 + ri * 9 + k0 + lane;
                const int up[3] = {1, 2, 5}, low[3] = {3, 6, 7};
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    const double a = v[(int64_t)up[u] * ni], b = v[(int64_t)low[u] * ni];
                    if (__double_as_longlong(a) == __double_as_longlong(b)) continue;
                    double d = 0.0;
                    for (int e = 0; e < 9; e += 4) d = fmax(d, fabs(v[(int64_t)e * ni]));
                    if (!(fabs(a - b) <= 1e-9 * fmax(fabs(a), fabs(b)) + 1e-12 * d)) *skew = 1ull;
                }
            }
            unsigned todo = __ballot_sync(0xffffffffu, mine > i);
            while (todo) {
                int at[3], to[3], slot[3], len[3];
                int64_t start[3];
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    at[u] = todo ? __ffs(todo) - 1 : -1;
                    todo &= todo - 1;
                    to[u] = __shfl_sync(0xffffffffu, mine, max(at[u], 0));
                    const int64_t j = at[u] >= 0 ? to[u] : i;
                    start[u] = rp[j];
                    len[u] = (int)(rp[j + 1] - start[u]);
                }
                int first[3];
#pragma unroll
                for (int u = 0; u < 3; ++u) first[u] = lane < len[u] ? bcol[start[u] + lane] : -1;
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    unsigned hit = __ballot_sync(0xffffffffu, first[u] == i);
                    slot[u] = hit ? __ffs(hit) - 1 : -1;
                    for (int q0 = 32; slot[u] < 0 && q0 < len[u]; q0 += 32) {
                        hit = __ballot_sync(0xffffffffu, q0 + lane < len[u] && bcol[start[u] + q0 + lane] == i);
                        if (hit) slot[u] = q0 + __ffs(hit) - 1;
                    }
                    if (at[u] >= 0 && slot[u] < 0) ++nbad;  // no partner
                }
                const int64_t st3 = u3 == 0 ? start[0] : (u3 == 1 ? start[1] : start[2]);
                const int ln3 = u3 == 0 ? len[0] : (u3 == 1 ? len[1] : len[2]);
                const int sl3 = u3 == 0 ? slot[0] : (u3 == 1 ? slot[1] : slot[2]);
                const int at3 = u3 == 0 ? at[0] : (u3 == 1 ? at[1] : at[2]);
                const bool have = lane < 27 && at3 >= 0 && sl3 >= 0;
                double a = 0.0, b = 0.0;
                if (have) {
                    a = v64[ri * 9 + (int64_t)e3 * ni + k0 + at3];
                    b = v64[st3 * 9 + (int64_t)(3 * c3 + r3) * ln3 + sl3];
                }
                // (equal bits of an infinity or a NaN are no agreement)
                const bool differ = have && (__double_as_longlong(a) != __double_as_longlong(b) ||
                                             (__double2hiint(a) & 0x7ff00000) == 0x7ff00000);
                if (__any_sync(0xffffffffu, differ)) {
                    const double di = diag_scale(i);
                    double dj = 0.0;
#pragma unroll
                    for (int u = 0; u < 3; ++u) {
                        const double d = diag_scale(at[u] >= 0 ? to[u] : i);
                        if (u == u3) dj = d;
                    }
                    const bool ok = !differ || fabs(a - b) <= 1e-9 * fmax(fabs(a), fabs(b)) + 1e-12 * fmax(di, dj);
                    const unsigned no = __ballot_sync(0xffffffffu, !ok);
                    nbad += ((no & 0x1ffu) != 0) + ((no & 0x3fe00u) != 0) + ((no & 0x7fc0000u) != 0);
                }
            }
        }
        if (nbad && lane == 0) atomicAdd(bad, nbad);
    }
}

// max over scalar rows of sum_j |a_ij| (as FP32 bits), a warp per block row:
// the bound the fixed-point symmetric product sizes its quantum from.
__global__ void k_rowsum_max(int64_t nb, const int64_t *__restrict__ rp, const double *__restrict__ v64,
                             unsigned *__restrict__ out)
{
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    float best = 0.f;
    for (int64_t i = w0; i < nb; i += nw) {
        const int64_t r0 = rp[i];
        const int n = (int)(rp[i + 1] - r0);
        float sum[3] = {0.f, 0.f, 0.f};
        for (int k = lane; k < n; k += 32)
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c) sum[r] += fabsf((float)v64[r0 * 9 + (int64_t)(3 * r + c) * n + k]);
#pragma unroll
        for (int r = 0; r < 3; ++r) best = fmaxf(best, warp_sum(sum[r]));
    }
    if (lane == 0) atomicMax(out, __float_as_uint(best));
}

void check_symmetric(DevMatrix &A, cudaStream_t st)
{
    PFG_CHECK(A.nb > 0, PFG_E_STATE, "empty matrix");
    PFG_CHECK(A.bs == 3, PFG_E_UNSUPPORTED, "symmetric storage is built for 3x3-block matrices");
    if (A.sym_checked) return;
    // the values (pattern included) changed: check the symmetry once
    DevBuf<unsigned long long> bad(2);  // pairs that differ; whether a diagonal block does
    PFG_CUDA(cudaMemsetAsync(bad.p, 0, 2 * sizeof(unsigned long long), st));
    k_sym_check<<<grid_for(A.nb, 8, sm_count_device() * 16), 256, 0, st>>>(A.nb, A.rp.p, A.col.p, A.v64.p, bad.p,
                                                                           bad.p + 1);
    PFG_CUDA(cudaGetLastError());
    unsigned long long found[2] = {0, 0};
    PFG_CUDA(cudaMemcpyAsync(found, bad.p, sizeof found, cudaMemcpyDeviceToHost, st));
    PFG_CUDA(cudaStreamSynchronize(st));
    PFG_CHECK(found[0] == 0, PFG_E_ARG,
              "symmetric storage needs a symmetric matrix: " + std::to_string(found[0]) +
                  " blocks differ from their transposes");
    A.skew_diagonal = found[1] != 0;
    A.sym_checked = true;
}

void bound_rows(DevMatrix &A, cudaStream_t st)
{
    if (A.sym_rowsum_valid) return;
    DevBuf<unsigned> bits(1);
    PFG_CUDA(cudaMemsetAsync(bits.p, 0, sizeof(unsigned), st));
    k_rowsum_max<<<grid_for(A.nb, 8, sm_count_device() * 16), 256, 0, st>>>(A.nb, A.rp.p, A.v64.p, bits.p);
    PFG_CUDA(cudaGetLastError());
    PFG_CUDA(cudaMemcpyAsync(&A.sym_rowsum, bits.p, sizeof(float), cudaMemcpyDeviceToHost, st));
    PFG_CUDA(cudaStreamSynchronize(st));
    A.sym_rowsum_valid = true;
}

void build_sell_upper(DevMatrix &A, cudaStream_t st)
{
    check_symmetric(A, st);
    if (A.sell_u_pattern && A.s32_u_valid) return;
    if (!A.sell_u_pattern) {
        A.ns_u = (A.nb + 31) / 32;
        DevBuf<int64_t> width((size_t)A.ns_u + 1);
        PFG_CUDA(cudaMemsetAsync(width.p, 0, (A.ns_u + 1) * sizeof(int64_t), st));
        k_sellu_widths<<<grid_for(A.ns_u, 256, sm_count_device() * 16), 256, 0, st>>>(A.nb, A.ns_u, A.rp.p, A.col.p, width.p);
        PFG_CUDA(cudaGetLastError());
        A.sptr_u.resize((size_t)A.ns_u + 1);
        const int64_t slots = exclusive_scan(width.p, A.sptr_u.p, A.ns_u + 1, st);
        A.scol_u.resize((size_t)std::max<int64_t>(slots * 32, 1));
        A.s32_u.resize((size_t)std::max<int64_t>(slots * 32 * 9, 1));
        A.sell_u_pattern = true;
    }
    k_sellu_fill<<<(int)std::min<int64_t>(A.ns_u, sm_count_device() * 16), 288, 0, st>>>(
        A.nb, A.ns_u, A.rp.p, A.col.p, A.v64.p, A.sptr_u.p, A.scol_u.p, A.s32_u.p);
    PFG_CUDA(cudaGetLastError());
    A.s32_u_valid = true;
}

}  // namespace pfg
