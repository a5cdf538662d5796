// lobpcg.cu -- block LOBPCG on the device (see lobpcg.cuh).
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "lobpcg.cuh"

namespace pfg {

// ===================================================================== host
// Symmetric eigensolver for the small Rayleigh-Ritz problems: Householder
// reduction to tridiagonal form with accumulated transformations, then the
// implicit QL iteration with shifts (Bowdler, Martin, Reinsch & Wilkinson,
// Numer. Math. 11 (1968), the method of EISPACK's tql2).  A is n x n column-
// major, replaced by the eigenvectors; w receives the eigenvalues ascending.
static void sym_eig(int n, std::vector<double> &A, std::vector<double> &w)
{
    auto a = [&](int i, int j) -> double & { return A[(size_t)j * n + i]; };
    std::vector<double> Q((size_t)n * n, 0.0), d(n), e(n, 0.0), v(n), p(n), q(n);
    for (int i = 0; i < n; ++i) Q[(size_t)i * n + i] = 1.0;
    // Householder: zero column j below the subdiagonal
    for (int j = 0; j + 2 < n; ++j) {
        double alpha = 0.0;
        for (int i = j + 1; i < n; ++i) alpha += a(i, j) * a(i, j);
        alpha = std::sqrt(alpha);
        if (alpha == 0.0) continue;
        if (a(j + 1, j) > 0) alpha = -alpha;
        // v = x - alpha e1 on rows j+1..n-1
        for (int i = 0; i < n; ++i) v[i] = 0.0;
        for (int i = j + 1; i < n; ++i) v[i] = a(i, j);
        v[j + 1] -= alpha;
        double vv = 0.0;
        for (int i = j + 1; i < n; ++i) vv += v[i] * v[i];
        if (vv == 0.0) continue;
        const double beta = 2.0 / vv;
        // A <- H A H with H = I - beta v v^T:  p = beta A v, K = beta/2 v^T p, q = p - K v,
        // A <- A - v q^T - q v^T.  Columns < j are reduced already (zero below
        // their subdiagonal), so p, q and the update live in rows/columns >= j.
        for (int i = j; i < n; ++i) {
            double s = 0.0;
            for (int l = j + 1; l < n; ++l) s += a(i, l) * v[l];
            p[i] = beta * s;
        }
        double K = 0.0;
        for (int i = j + 1; i < n; ++i) K += v[i] * p[i];
        K *= 0.5 * beta;
        for (int i = j; i < n; ++i) q[i] = p[i] - K * v[i];
        for (int c = j; c < n; ++c)
            for (int r = j; r < n; ++r) a(r, c) -= v[r] * q[c] + q[r] * v[c];
        // Q <- Q H = Q - beta (Q v) v^T, column by column (contiguous)
        for (int r = 0; r < n; ++r) p[r] = 0.0;
        for (int l = j + 1; l < n; ++l) {
            const double vl = v[l];
            const double *ql = &Q[(size_t)l * n];
            for (int r = 0; r < n; ++r) p[r] += ql[r] * vl;
        }
        for (int l = j + 1; l < n; ++l) {
            const double bv = beta * v[l];
            double *ql = &Q[(size_t)l * n];
            for (int r = 0; r < n; ++r) ql[r] -= p[r] * bv;
        }
    }
    for (int i = 0; i < n; ++i) d[i] = a(i, i);
    for (int i = 0; i + 1 < n; ++i) e[i] = a(i + 1, i);
    e[n - 1] = 0.0;
    // implicit QL on (d, e), rotations applied to the columns of Q
    const double eps = 2.220446049250313e-16;
    for (int l = 0; l < n; ++l) {
        for (int iter = 0; iter < 200; ++iter) {
            int m = l;
            for (; m < n - 1; ++m) {
                const double dd = std::fabs(d[m]) + std::fabs(d[m + 1]);
                if (std::fabs(e[m]) <= eps * dd) break;
            }
            if (m == l) break;
            // sqrt(x*x + y*y) in place of hypot: the matrices are scaled to
            // unit diagonal (B) or come from it (A'), far from overflow
            double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
            double r = std::sqrt(g * g + 1.0);
            g = d[m] - d[l] + e[l] / (g + (g >= 0 ? r : -r));
            double s = 1.0, c = 1.0, pp = 0.0;
            int i = m - 1;
            bool underflow = false;
            for (; i >= l; --i) {
                const double f = s * e[i], b = c * e[i];
                r = std::sqrt(f * f + g * g);
                e[i + 1] = r;
                if (r == 0.0) {
                    d[i + 1] -= pp;
                    e[m] = 0.0;
                    underflow = true;
                    break;
                }
                s = f / r;
                c = g / r;
                g = d[i + 1] - pp;
                r = (d[i] - g) * s + 2.0 * c * b;
                pp = s * r;
                d[i + 1] = g + pp;
                g = c * r - b;
                double *qi = &Q[(size_t)i * n], *qi1 = &Q[(size_t)(i + 1) * n];
                for (int k = 0; k < n; ++k) {
                    const double t = qi1[k];
                    qi1[k] = s * qi[k] + c * t;
                    qi[k] = c * qi[k] - s * t;
                }
            }
            if (underflow) continue;
            d[l] -= pp;
            e[l] = g;
            e[m] = 0.0;
        }
    }
    // sort ascending
    std::vector<int> idx(n);
    for (int i = 0; i < n; ++i) idx[i] = i;
    std::sort(idx.begin(), idx.end(), [&](int x, int y) { return d[x] < d[y]; });
    w.assign(n, 0.0);
    for (int i = 0; i < n; ++i) {
        w[i] = d[idx[i]];
        for (int r = 0; r < n; ++r) A[(size_t)i * n + r] = Q[(size_t)idx[i] * n + r];
    }
}

// The lowest k eigenpairs of a symmetric A (n x n, column-major; destroyed):
// Householder reduction to tridiagonal T = Q^T A Q without accumulating Q,
// T's eigenvalues by the implicit QL iteration without vectors (tql1), the k
// wanted eigenvectors of T by inverse iteration (Peters & Wilkinson, "The
// calculation of specified eigenvectors by inverse iteration", Handbook for
// Automatic Computation II (1971); the scheme of LAPACK's dstein: tridiagonal
// LU with partial pivoting, tiny pivots replaced by eps ||T||, shifts of
// coincident eigenvalues spread by 10 eps ||T||, modified Gram-Schmidt against
// the earlier vectors of a cluster, i.e. of eigenvalues within 1e-3 ||T||),
// and the back transformation Q y by the stored reflectors.  About a third of
// the work of sym_eig at n = 72, k = 24 (no n x n accumulation of Q).
// w: all n eigenvalues ascending; Y: n x k, column j the eigenvector of w[j].
static void sym_eig_lowest(int n, std::vector<double> &A, int k, std::vector<double> &w, std::vector<double> &Y)
{
    auto a = [&](int i, int j) -> double & { return A[(size_t)j * n + i]; };
    std::vector<double> d(n), e(n, 0.0), V((size_t)n * n, 0.0), beta(n, 0.0), v(n), p(n), q(n);
    for (int j = 0; j + 2 < n; ++j) {
        double alpha = 0.0;
        for (int i = j + 1; i < n; ++i) alpha += a(i, j) * a(i, j);
        alpha = std::sqrt(alpha);
        if (alpha == 0.0) continue;
        if (a(j + 1, j) > 0) alpha = -alpha;
        for (int i = 0; i < n; ++i) v[i] = 0.0;
        for (int i = j + 1; i < n; ++i) v[i] = a(i, j);
        v[j + 1] -= alpha;
        double vv = 0.0;
        for (int i = j + 1; i < n; ++i) vv += v[i] * v[i];
        if (vv == 0.0) continue;
        const double bt = 2.0 / vv;
        // p = beta A v as a sum of columns (contiguous, vectorisable loops)
        for (int i = j; i < n; ++i) p[i] = 0.0;
        for (int l = j + 1; l < n; ++l) {
            const double vl = bt * v[l];
            const double *al = &A[(size_t)l * n];
            for (int i = j; i < n; ++i) p[i] += al[i] * vl;
        }
        double K = 0.0;
        for (int i = j + 1; i < n; ++i) K += v[i] * p[i];
        K *= 0.5 * bt;
        for (int i = j; i < n; ++i) q[i] = p[i] - K * v[i];
        for (int c = j; c < n; ++c)
            for (int r = j; r < n; ++r) a(r, c) -= v[r] * q[c] + q[r] * v[c];
        for (int i = j + 1; i < n; ++i) V[(size_t)j * n + i] = v[i];
        beta[j] = bt;
    }
    double tnorm = 0.0;
    for (int i = 0; i < n; ++i) {
        d[i] = a(i, i);
        if (i + 1 < n) e[i] = a(i + 1, i);
    }
    for (int i = 0; i < n; ++i)
        tnorm = std::max(tnorm, std::fabs(d[i]) + (i > 0 ? std::fabs(e[i - 1]) : 0.0) + std::fabs(e[i]));
    // eigenvalues: implicit QL on copies of (d, e), no vectors
    const double eps = 2.220446049250313e-16;
    {
        std::vector<double> dd = d, ee = e;
        ee[n - 1] = 0.0;
        for (int l = 0; l < n; ++l) {
            for (int iter = 0; iter < 200; ++iter) {
                int m = l;
                for (; m < n - 1; ++m) {
                    const double s = std::fabs(dd[m]) + std::fabs(dd[m + 1]);
                    if (std::fabs(ee[m]) <= eps * s) break;
                }
                if (m == l) break;
                double g = (dd[l + 1] - dd[l]) / (2.0 * ee[l]);
                double r = std::sqrt(g * g + 1.0);
                g = dd[m] - dd[l] + ee[l] / (g + (g >= 0 ? r : -r));
                double s = 1.0, c = 1.0, pp = 0.0;
                bool underflow = false;
                for (int i = m - 1; i >= l; --i) {
                    const double f = s * ee[i], b = c * ee[i];
                    r = std::sqrt(f * f + g * g);
                    ee[i + 1] = r;
                    if (r == 0.0) {
                        dd[i + 1] -= pp;
                        ee[m] = 0.0;
                        underflow = true;
                        break;
                    }
                    s = f / r;
                    c = g / r;
                    g = dd[i + 1] - pp;
                    r = (dd[i] - g) * s + 2.0 * c * b;
                    pp = s * r;
                    dd[i + 1] = g + pp;
                    g = c * r - b;
                }
                if (underflow) continue;
                dd[l] -= pp;
                ee[l] = g;
                ee[m] = 0.0;
            }
        }
        std::sort(dd.begin(), dd.end());
        w = dd;
    }
    // inverse iteration for the k lowest
    const int kk = std::min(k, n);
    Y.assign((size_t)n * kk, 0.0);
    const double tiny = eps * std::max(tnorm, 1e-300);
    const double ortol = 1e-3 * tnorm, pertol = 10.0 * eps * tnorm;
    std::vector<double> dl(n), dg(n), du(n), du2(n), x(n), Yt((size_t)n * kk);  // Yt: T's eigenvectors
    std::vector<char> piv(n);
    int cluster0 = 0;
    double prev = 0.0;
    for (int j = 0; j < kk; ++j) {
        double lam = w[j];
        if (j > 0) {
            if (w[j] - w[j - 1] > ortol) cluster0 = j;
            if (lam <= prev + pertol) lam = prev + pertol;  // distinct shifts inside a cluster
        }
        prev = lam;
        // LU of T - lam I with partial pivoting (U: diagonal dg, superdiagonals du, du2)
        for (int i = 0; i < n; ++i) {
            dg[i] = d[i] - lam;
            dl[i] = du[i] = (i + 1 < n) ? e[i] : 0.0;
            du2[i] = 0.0;
        }
        for (int i = 0; i + 1 < n; ++i) {
            if (std::fabs(dg[i]) >= std::fabs(dl[i])) {
                piv[i] = 0;
                if (std::fabs(dg[i]) < tiny) dg[i] = dg[i] < 0 ? -tiny : tiny;
                const double f = dl[i] / dg[i];
                dl[i] = f;
                dg[i + 1] -= f * du[i];
            } else {
                piv[i] = 1;
                const double f = dg[i] / dl[i];
                dg[i] = dl[i];
                dl[i] = f;
                const double t = du[i];
                du[i] = dg[i + 1];
                dg[i + 1] = t - f * dg[i + 1];
                if (i + 2 < n) {
                    du2[i] = du[i + 1];
                    du[i + 1] = -f * du[i + 1];
                }
            }
        }
        if (std::fabs(dg[n - 1]) < tiny) dg[n - 1] = dg[n - 1] < 0 ? -tiny : tiny;
        for (int i = 0; i < n; ++i) dg[i] = 1.0 / dg[i];  // pivots kept as reciprocals for the solves
        // start: a fixed pseudo-random vector (different per j)
        for (int i = 0; i < n; ++i) {
            uint64_t h = (uint64_t)(j + 1) * 0x9e3779b97f4a7c15ull ^ ((uint64_t)i * 0xbf58476d1ce4e5b9ull);
            h ^= h >> 31;
            h *= 0x94d049bb133111ebull;
            h ^= h >> 29;
            x[i] = (double)(h >> 11) * (2.0 / 9007199254740992.0) - 1.0;
        }
        for (int it = 0; it < 3; ++it) {
            for (int i = 0; i + 1 < n; ++i) {  // L^-1 (with the row interchanges)
                if (piv[i]) std::swap(x[i], x[i + 1]);
                x[i + 1] -= dl[i] * x[i];
            }
            for (int i = n - 1; i >= 0; --i) {  // U^-1
                double t = x[i];
                if (i + 1 < n) t -= du[i] * x[i + 1];
                if (i + 2 < n) t -= du2[i] * x[i + 2];
                x[i] = t * dg[i];
            }
            for (int c = cluster0; c < j; ++c) {  // orthogonal to the cluster's earlier vectors
                const double *yc = &Yt[(size_t)c * n];
                double s = 0.0;
                for (int i = 0; i < n; ++i) s += yc[i] * x[i];
                for (int i = 0; i < n; ++i) x[i] -= s * yc[i];
            }
            double nrm = 0.0;
            for (int i = 0; i < n; ++i) nrm += x[i] * x[i];
            nrm = std::sqrt(nrm);
            if (!(nrm > 0.0) || !std::isfinite(nrm)) nrm = 1.0;
            for (int i = 0; i < n; ++i) x[i] /= nrm;
        }
        std::copy(x.begin(), x.end(), Yt.begin() + (size_t)j * n);
    }
    // back transformation of all kk vectors at once, y <- H_0 (H_1 (... (H_{n-3} y))):
    // the block is held row-major (n x kk), so each reflector's dot products
    // and updates run along contiguous rows of kk values
    std::vector<double> Xr((size_t)n * kk), sv(kk);
    for (int c = 0; c < kk; ++c)
        for (int i = 0; i < n; ++i) Xr[(size_t)i * kk + c] = Yt[(size_t)c * n + i];
    for (int jj = n - 3; jj >= 0; --jj) {
        if (beta[jj] == 0.0) continue;
        const double *vj = &V[(size_t)jj * n];
        for (int c = 0; c < kk; ++c) sv[c] = 0.0;
        for (int i = jj + 1; i < n; ++i) {
            const double vi = vj[i];
            const double *xi = &Xr[(size_t)i * kk];
            for (int c = 0; c < kk; ++c) sv[c] += vi * xi[c];
        }
        for (int c = 0; c < kk; ++c) sv[c] *= beta[jj];
        for (int i = jj + 1; i < n; ++i) {
            const double vi = vj[i];
            double *xi = &Xr[(size_t)i * kk];
            for (int c = 0; c < kk; ++c) xi[c] -= sv[c] * vi;
        }
    }
    for (int c = 0; c < kk; ++c)
        for (int i = 0; i < n; ++i) Y[(size_t)c * n + i] = Xr[(size_t)i * kk + c];
}

// B = L L^T (lower L, column-major, in place of B's lower triangle) when every
// pivot exceeds rank_tol times the largest diagonal entry; false otherwise.
static bool cholesky_well_posed(int m, std::vector<double> &B, double rank_tol)
{
    double dmax = 0.0;
    for (int i = 0; i < m; ++i) dmax = std::max(dmax, B[(size_t)i * m + i]);
    if (!(dmax > 0.0)) return false;
    // right-looking: scale column j, then update the trailing columns (each
    // update a contiguous column axpy)
    for (int j = 0; j < m; ++j) {
        double *bj = &B[(size_t)j * m];
        const double d = bj[j];
        if (!(d > rank_tol * dmax)) return false;
        const double ljj = std::sqrt(d);
        bj[j] = ljj;
        const double inv = 1.0 / ljj;
        for (int i = j + 1; i < m; ++i) bj[i] *= inv;
        for (int c = j + 1; c < m; ++c) {
            double *bc = &B[(size_t)c * m];
            const double f = bj[c];
            for (int i = c; i < m; ++i) bc[i] -= bj[i] * f;
        }
    }
    return true;
}

int small_generalized_eig(int m, const double *Ain, const double *Bin, int k, double rank_tol, double *lam, double *C)
{
    // scale to unit diagonal, then keep B's numerically nonzero directions
    std::vector<double> s(m);
    for (int i = 0; i < m; ++i) {
        const double b = Bin[(size_t)i * m + i];
        s[i] = (b > 0 && std::isfinite(b)) ? 1.0 / std::sqrt(b) : 0.0;
    }
    std::vector<double> B((size_t)m * m), w;
    for (int j = 0; j < m; ++j)
        for (int i = 0; i < m; ++i)
            B[(size_t)j * m + i] = 0.5 * (Bin[(size_t)j * m + i] + Bin[(size_t)i * m + j]) * s[i] * s[j];
    {
        // Well-posed B (no pivot at or below rank_tol of the largest: the
        // usual case): A' = L^-1 (S A S) L^-T and C = S L^-T Y, a Cholesky
        // and two triangular solves instead of B's eigendecomposition.
        // Otherwise B's eigendecomposition below drops its null directions.
        std::vector<double> L = B;
        if (cholesky_well_posed(m, L, rank_tol)) {
            // Block forward substitution X <- L^-1 X on a row-major m x w
            // block: each step scales row q and subtracts it from the rows
            // below, whole rows at a time (contiguous, vectorisable).
            auto block_lsolve = [&](double *X, int w) {
                for (int q = 0; q < m; ++q) {
                    const double *lq = &L[(size_t)q * m];  // column q of L
                    double *xq = X + (size_t)q * w;
                    const double inv = 1.0 / lq[q];
                    for (int c = 0; c < w; ++c) xq[c] *= inv;
                    for (int i = q + 1; i < m; ++i) {
                        const double f = lq[i];
                        double *xi = X + (size_t)i * w;
                        for (int c = 0; c < w; ++c) xi[c] -= f * xq[c];
                    }
                }
            };
            // W = L^-1 (S A S); A' = W L^-T = (L^-1 W^T)^T (symmetric)
            std::vector<double> W((size_t)m * m), Ap((size_t)m * m);
            for (int r = 0; r < m; ++r)
                for (int c = 0; c < m; ++c)
                    W[(size_t)r * m + c] = 0.5 * (Ain[(size_t)c * m + r] + Ain[(size_t)r * m + c]) * s[r] * s[c];
            block_lsolve(W.data(), m);
            for (int r = 0; r < m; ++r)
                for (int c = 0; c < m; ++c) Ap[(size_t)r * m + c] = W[(size_t)c * m + r];
            block_lsolve(Ap.data(), m);
            for (int c = 0; c < m; ++c)  // symmetrise
                for (int r = 0; r < c; ++r) {
                    const double v = 0.5 * (Ap[(size_t)c * m + r] + Ap[(size_t)r * m + c]);
                    Ap[(size_t)c * m + r] = Ap[(size_t)r * m + c] = v;
                }
            std::vector<double> mu, Y;
            const int kk = std::min(k, m);
            sym_eig_lowest(m, Ap, kk, mu, Y);
            // C = S L^-T Y: block back substitution on the row-major m x kk
            // block of the eigenvectors
            std::vector<double> Cb((size_t)m * kk);
            for (int j2 = 0; j2 < kk; ++j2)
                for (int r = 0; r < m; ++r) Cb[(size_t)r * kk + j2] = Y[(size_t)j2 * m + r];
            for (int r = m - 1; r >= 0; --r) {
                double *cr = &Cb[(size_t)r * kk];
                const double inv = 1.0 / L[(size_t)r * m + r];
                for (int c = 0; c < kk; ++c) cr[c] *= inv;
                for (int q = 0; q < r; ++q) {
                    const double f = L[(size_t)q * m + r];  // L(r, q) = L^T(q, r)
                    double *cq = &Cb[(size_t)q * kk];
                    for (int c = 0; c < kk; ++c) cq[c] -= f * cr[c];
                }
            }
            for (int j2 = 0; j2 < kk; ++j2) {
                lam[j2] = mu[j2];
                for (int r = 0; r < m; ++r) C[(size_t)j2 * m + r] = Cb[(size_t)r * kk + j2] * s[r];
            }
            return kk;
        }
    }
    sym_eig(m, B, w);
    const double wmax = w[m - 1];
    if (!(wmax > 0)) return 0;
    std::vector<int> keep;
    for (int i = 0; i < m; ++i)
        if (w[i] > rank_tol * wmax) keep.push_back(i);
    const int r = (int)keep.size();
    // T = S Q_keep Theta^-1/2  (m x r)
    std::vector<double> T((size_t)m * r);
    for (int c = 0; c < r; ++c) {
        const double f = 1.0 / std::sqrt(w[keep[c]]);
        for (int i = 0; i < m; ++i) T[(size_t)c * m + i] = s[i] * B[(size_t)keep[c] * m + i] * f;
    }
    // A' = T^T A T
    std::vector<double> AT((size_t)m * r), Ap((size_t)r * r);
    for (int c = 0; c < r; ++c)
        for (int i = 0; i < m; ++i) {
            double acc = 0.0;
            for (int l = 0; l < m; ++l) acc += 0.5 * (Ain[(size_t)l * m + i] + Ain[(size_t)i * m + l]) * T[(size_t)c * m + l];
            AT[(size_t)c * m + i] = acc;
        }
    for (int c = 0; c < r; ++c)
        for (int i = 0; i < r; ++i) {
            double acc = 0.0;
            for (int l = 0; l < m; ++l) acc += T[(size_t)i * m + l] * AT[(size_t)c * m + l];
            Ap[(size_t)c * r + i] = acc;
        }
    for (int c = 0; c < r; ++c)
        for (int i = 0; i < c; ++i) {
            const double v = 0.5 * (Ap[(size_t)c * r + i] + Ap[(size_t)i * r + c]);
            Ap[(size_t)c * r + i] = Ap[(size_t)i * r + c] = v;
        }
    std::vector<double> mu;
    sym_eig(r, Ap, mu);
    const int kk = std::min(k, r);
    for (int j = 0; j < kk; ++j) {
        lam[j] = mu[j];
        for (int i = 0; i < m; ++i) {
            double acc = 0.0;
            for (int l = 0; l < r; ++l) acc += T[(size_t)l * m + i] * Ap[(size_t)j * r + l];
            C[(size_t)j * m + i] = acc;
        }
    }
    return kk;
}

// =================================================================== device
constexpr int kT = 256;
constexpr int PW = 8;  // panel width

template <typename T>
__device__ __forceinline__ const T *panel_row(const T *base, int64_t n, int q, int64_t row)
{
    return base + ((int64_t)q * n + row) * PW;
}

// A panel row (PW = 8 consecutive values, 32 or 64 bytes, aligned to its
// size) moved with 16-byte accesses: one gather instruction per 16 bytes
// instead of one per value.
__device__ __forceinline__ void ld_row(const float *p, float (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const float4 w = __ldg(reinterpret_cast<const float4 *>(p) + u);
        v[4 * u] = w.x;
        v[4 * u + 1] = w.y;
        v[4 * u + 2] = w.z;
        v[4 * u + 3] = w.w;
    }
}
__device__ __forceinline__ void ld_row(const double *p, double (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const double2 w = __ldg(reinterpret_cast<const double2 *>(p) + u);
        v[2 * u] = w.x;
        v[2 * u + 1] = w.y;
    }
}
__device__ __forceinline__ void ld_row(const float2 *p, float2 (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const float4 w = __ldg(reinterpret_cast<const float4 *>(p) + u);
        v[2 * u] = make_float2(w.x, w.y);
        v[2 * u + 1] = make_float2(w.z, w.w);
    }
}
__device__ __forceinline__ void st_row(float *p, const float (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < 2; ++u)
        reinterpret_cast<float4 *>(p)[u] = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
}
__device__ __forceinline__ void st_row(double *p, const double (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < 4; ++u) reinterpret_cast<double2 *>(p)[u] = make_double2(v[2 * u], v[2 * u + 1]);
}
__device__ __forceinline__ void st_row(float2 *p, const float2 (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < 4; ++u)
        reinterpret_cast<float4 *>(p)[u] = make_float4(v[2 * u].x, v[2 * u].y, v[2 * u + 1].x, v[2 * u + 1].y);
}
// The same from shared memory (plain loads: __ldg is for global memory).
__device__ __forceinline__ void lds_row(const float *p, float (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const float4 w = reinterpret_cast<const float4 *>(p)[u];
        v[4 * u] = w.x;
        v[4 * u + 1] = w.y;
        v[4 * u + 2] = w.z;
        v[4 * u + 3] = w.w;
    }
}
__device__ __forceinline__ void lds_row(const double *p, double (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const double2 w = reinterpret_cast<const double2 *>(p)[u];
        v[2 * u] = w.x;
        v[2 * u + 1] = w.y;
    }
}

// Double-FP32 ("double-float") arithmetic on the FP32 pipe, for the second
// phase of the mixed LOBPCG (its Gram, SpMM and linear combinations of FP64
// panels): GB300's FP64 pipe is about 1/30 of its FP32 pipe, and the FP64
// forms of these kernels ran on it (the Gram at 0.92 TFLOP/s).  Each FP64 value is split into hi + lo floats (exact to
// 48 bits); a product's rounding error comes exactly from an FMA (Dekker's
// product), the cross terms hi*lo are added to it, and each sum keeps its
// rounding error by TwoSum (Knuth); the pair (hi, lo) accumulates one CTA's
// rows and the partial sums are added in FP64 (Hida, Li & Bailey 2001, "Algorithms
// for quad-double precision", double-double addition and multiplication).
// Explicit _rn intrinsics keep the compiler from contracting the error-free
// steps into FMAs.  Relative error about n_cta * 2^-48 per partial sum.
struct DFAcc {
    float hi, lo;
    __device__ void zero() { hi = lo = 0.f; }
    __device__ void add(float2 a, float2 b)
    {
        const float p = __fmul_rn(a.x, b.x);
        float e = fmaf(a.x, b.x, -p);
        e = fmaf(a.x, b.y, e);
        e = fmaf(a.y, b.x, e);
        const float t = __fadd_rn(hi, p);
        const float z = __fsub_rn(t, hi);
        const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(t, z)), __fsub_rn(p, z));
        hi = t;
        lo = __fadd_rn(lo, __fadd_rn(err, e));
    }
    __device__ double get() const { return (double)hi + (double)lo; }
    // the sum as a normalised (hi, lo) pair: TwoSum of the two parts (FP32 only)
    __device__ float2 get2() const
    {
        const float s = __fadd_rn(hi, lo);
        const float z = __fsub_rn(s, hi);
        return make_float2(s, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, z)), __fsub_rn(lo, z)));
    }
};

// Two FP32 values in one 64-bit register pair: add, mul and fma.rn.f32x2 work on
// both.  The pipe does no more of them per clock than of the scalar forms (measured
// 128 values per clock and SM either way), but in half the issue slots and fewer
// registers: linear combinations 996 -> 852 us at 398k rows and 24 columns, 78 -> 56
// at 70k and 12 (where the half panel counts too), the Gram matrices 104 -> 94 there
// and 1,195 -> 1,177 at the larger size (pipe-bound at 12 operations a multiply-add).
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2_pack(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2_get(F2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Two DFAcc side by side, the same operations in the same order (a subtraction as an
// FMA by -1, which rounds once just so): the same bits.  a is common to both.
struct DFLeft {  // a double-float factor and its negated head, each twice
    F2 h, nh, l;
    __device__ explicit DFLeft(float2 a) : h(f2_pack(a.x, a.x)), nh(f2_pack(-a.x, -a.x)), l(f2_pack(a.y, a.y)) {}
};
struct DFAcc2 {
    F2 hi, lo;
    __device__ void zero() { hi = lo = 0ull; }
    __device__ void add(const DFLeft &a, F2 bh, F2 bl)
    {
        const F2 m1 = 0xbf800000bf800000ull;  // (-1, -1)
        const F2 np = f2_mul(a.nh, bh);       // -p
        F2 e = f2_fma(a.h, bh, np);
        e = f2_fma(a.h, bl, e);
        e = f2_fma(a.l, bh, e);
        const F2 t = f2_fma(np, m1, hi);
        const F2 z = f2_fma(hi, m1, t);
        const F2 u = f2_fma(f2_fma(z, m1, t), m1, hi);  // hi - (t - z)
        const F2 err = f2_fma(f2_add(np, z), m1, u);    // + (p - z)
        hi = t;
        lo = f2_add(lo, f2_add(err, e));
    }
    __device__ DFAcc get(int c) const
    {
        const float2 h = f2_get(hi), l = f2_get(lo);
        DFAcc r;
        r.hi = c ? h.y : h.x;
        r.lo = c ? l.y : l.x;
        return r;
    }
};

// Eight double-float values, heads and tails in pairs of columns, and the sums of
// a x row over them.  (The sliced products keep DFAcc: their rows come one by one
// from L2, and packed they took 571 us where DFAcc takes 465.)
struct DFRow {
    F2 h[PW / 2], l[PW / 2];
    template <int NC>
    __device__ void load_paired(const float2 *p)  // shared memory: two heads, two tails
    {
#pragma unroll
        for (int u = 0; u < NC / 2; ++u) {
            const ulonglong2 w = reinterpret_cast<const ulonglong2 *>(p)[u];
            h[u] = w.x;
            l[u] = w.y;
        }
    }
};
struct DFRowAcc {
    DFAcc2 v[PW / 2];
    __device__ void zero()
    {
#pragma unroll
        for (int u = 0; u < PW / 2; ++u) v[u].zero();
    }
    template <int NC>
    __device__ void add(float2 a, const DFRow &x)
    {
        const DFLeft f(a);
#pragma unroll
        for (int u = 0; u < NC / 2; ++u) v[u].add(f, x.h[u], x.l[u]);
    }
    __device__ float2 get(int c) const { return v[c >> 1].get(c & 1).get2(); }
};

__device__ __forceinline__ float2 df_split(double x)
{
    const float h = __double2float_rn(x);
    return make_float2(h, __double2float_rn(x - (double)h));
}

__device__ __forceinline__ double df_value(float2 v) { return (double)v.x + (double)v.y; }

// a + b of two double-float numbers (TwoSum of the heads, the tails added,
// renormalised by a second TwoSum)
__device__ __forceinline__ float2 df_add(float2 a, float2 b)
{
    const float s = __fadd_rn(a.x, b.x);
    const float z = __fsub_rn(s, a.x);
    float e = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, z)), __fsub_rn(b.x, z));
    e = __fadd_rn(e, __fadd_rn(a.y, b.y));
    const float t = __fadd_rn(s, e);
    const float z2 = __fsub_rn(t, s);
    return make_float2(t, __fadd_rn(__fsub_rn(s, __fsub_rn(t, z2)), __fsub_rn(e, z2)));
}

// The blocks of the iteration's three linear combinations (the vectors, their K and
// their M images): one launch, blockIdx.y picks.
template <typename T>
struct CombSet {
    const T *X[3], *W[3], *P[3];
    T *Xn[3], *Pn[3];
};

// Y = A X for every panel (one warp per (slice, panel), one lane per block
// row); rows of fixed DOFs are zeroed (the reduce_crs_matrix restriction).
template <int BS, typename T>
__global__ void __launch_bounds__(kT) k_spmm(SellView<T> A, int np, const T *__restrict__ X, T *__restrict__ Y,
                                             const uint8_t *__restrict__ fixed)
{
    const int lane = threadIdx.x & 31;
    const int64_t n = A.nb * BS;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t u = w0; u < A.ns * np; u += nw) {
        const int64_t s = u / np;
        const int q = (int)(u - s * np);
        const int64_t b0 = A.sptr[s];
        const int wdt = (int)(A.sptr[s + 1] - b0);
        const int *cp = A.col + b0 * 32 + lane;
        const T *vp = A.val + b0 * 32 * (BS * BS) + lane;
        T acc[BS][PW];
#pragma unroll
        for (int r = 0; r < BS; ++r)
#pragma unroll
            for (int c = 0; c < PW; ++c) acc[r][c] = T(0);
        for (int k = 0; k < wdt; ++k) {
            const int col = ld_stream(cp + (int64_t)k * 32);
            T a[BS * BS];
#pragma unroll
            for (int e = 0; e < BS * BS; ++e) a[e] = ld_stream(vp + ((int64_t)k * (BS * BS) + e) * 32);
#pragma unroll
            for (int cc = 0; cc < BS; ++cc) {
                T xv[PW];
                ld_row(panel_row(X, n, q, (int64_t)BS * col + cc), xv);
#pragma unroll
                for (int r = 0; r < BS; ++r)
#pragma unroll
                    for (int c = 0; c < PW; ++c) acc[r][c] = fma(a[r * BS + cc], xv[c], acc[r][c]);
            }
        }
        const int64_t row = s * 32 + lane;
        if (row < A.nb) {
#pragma unroll
            for (int r = 0; r < BS; ++r) {
                const int64_t i = (int64_t)BS * row + r;
                if (fixed && fixed[i])
#pragma unroll
                    for (int c = 0; c < PW; ++c) acc[r][c] = T(0);
                st_row(Y + ((int64_t)q * n + i) * PW, acc[r]);
            }
        }
    }
}

// ---- double-float forms of the SpMM and the linear combinations (mixed
// second phase).  That phase keeps its panels and images as (hi, lo) float
// pairs: the producers (SpMM, linear combinations, preconditioner, residual)
// write pairs, so the inner loops are FP32 arithmetic only and no conversion
// pass runs per iteration; only the matrices' FP64 values are split, once
// (k_to_df).  Splitting FP64 operands where they are used put a conversion
// per use on the FP64 pipe and was slower than FP64 itself; converting them
// in a pass before every use cost 16 % of a double-float iteration.
__global__ void k_to_df(int64_t len, const double *__restrict__ a, float2 *__restrict__ b)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = df_split(a[i]);
}

// Y = A X with A's sliced values (vdf, A's slot layout), the panels X and Y in
// double-float.  Layout and warp mapping as k_spmm.
template <int BS>
__global__ void __launch_bounds__(kT) k_spmm_df(SellView<double> A, const float2 *__restrict__ vdf, int np,
                                                const float2 *__restrict__ X, float2 *__restrict__ Y,
                                                const uint8_t *__restrict__ fixed)
{
    const int lane = threadIdx.x & 31;
    const int64_t n = A.nb * BS;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t u = w0; u < A.ns * np; u += nw) {
        const int64_t s = u / np;
        const int q = (int)(u - s * np);
        const int64_t b0 = A.sptr[s];
        const int wdt = (int)(A.sptr[s + 1] - b0);
        const int *cp = A.col + b0 * 32 + lane;
        const float2 *vp = vdf + b0 * 32 * (BS * BS) + lane;
        DFAcc acc[BS][PW];
#pragma unroll
        for (int r = 0; r < BS; ++r)
#pragma unroll
            for (int c = 0; c < PW; ++c) acc[r][c].zero();
        for (int k = 0; k < wdt; ++k) {
            const int col = ld_stream(cp + (int64_t)k * 32);
            float2 a[BS * BS];
#pragma unroll
            for (int e = 0; e < BS * BS; ++e) a[e] = __ldg(vp + ((int64_t)k * (BS * BS) + e) * 32);
#pragma unroll
            for (int cc = 0; cc < BS; ++cc) {
                float2 xv[PW];
                ld_row(panel_row(X, n, q, (int64_t)BS * col + cc), xv);
#pragma unroll
                for (int r = 0; r < BS; ++r)
#pragma unroll
                    for (int c = 0; c < PW; ++c) acc[r][c].add(a[r * BS + cc], xv[c]);
            }
        }
        const int64_t row = s * 32 + lane;
        if (row < A.nb) {
#pragma unroll
            for (int r = 0; r < BS; ++r) {
                const int64_t i = (int64_t)BS * row + r;
                const bool f = fixed && fixed[i];
                float2 yv[PW];
#pragma unroll
                for (int c = 0; c < PW; ++c) yv[c] = f ? make_float2(0.f, 0.f) : acc[r][c].get2();
                st_row(Y + ((int64_t)q * n + i) * PW, yv);
            }
        }
    }
}

// The products with kParts<T> warps per (slice, panel), each with a run of the
// slice's slots, the parts added in order: for systems whose slices and panels alone
// do not fill the GPU with warps.  A warp's slots are a chain of dependent loads (column,
// then three panel rows), 27 of them in a hex mesh: 49 us per launch at 23,247 block rows
// and two panels, whatever the bytes.  PAIR (FP32, K and M of one pattern): both
// products in one pass, so the columns and the panel rows, most of the traffic, are
// read once.  Measured there: K X and M X 94 -> 30 us (FP32; two parts 35, eight 42), one
// double-float product 96 -> 55 us (four parts 73, eight 83).
template <typename T>
constexpr int kParts = std::is_same<T, float2>::value ? 2 : 4;

template <typename T>
struct MulAcc;
template <>
struct MulAcc<float> {
    using Value = float;
    float v;
    __device__ void zero() { v = 0.f; }
    __device__ void add(float a, float x) { v = fmaf(a, x, v); }
    __device__ float get() const { return v; }
    __device__ static float sum(float a, float b) { return a + b; }
    __device__ static float none() { return 0.f; }
};
template <>
struct MulAcc<float2> {
    using Value = float2;
    DFAcc v;
    __device__ void zero() { v.zero(); }
    __device__ void add(float2 a, float2 x) { v.add(a, x); }
    __device__ float2 get() const { return v.get2(); }
    __device__ static float2 sum(float2 a, float2 b) { return df_add(a, b); }
    __device__ static float2 none() { return make_float2(0.f, 0.f); }
};

// the first NC columns of a panel row, 16 bytes a load
template <int NC>
__device__ __forceinline__ void ld_cols(const float *p, float (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < NC / 4; ++u) {
        const float4 w = __ldg(reinterpret_cast<const float4 *>(p) + u);
        v[4 * u] = w.x;
        v[4 * u + 1] = w.y;
        v[4 * u + 2] = w.z;
        v[4 * u + 3] = w.w;
    }
}
template <int NC>
__device__ __forceinline__ void ld_cols(const float2 *p, float2 (&v)[PW])
{
#pragma unroll
    for (int u = 0; u < NC / 2; ++u) {
        const float4 w = __ldg(reinterpret_cast<const float4 *>(p) + u);
        v[2 * u] = make_float2(w.x, w.y);
        v[2 * u + 1] = make_float2(w.z, w.w);
    }
}

// Slots [k0, k1) of a lane's row times the first NC columns of panel q.
template <int BS, int NC, typename T, int NM>
__device__ __forceinline__ void spmm_slots(int64_t b0, int k0, int k1, int lane, const int *__restrict__ scol,
                                           const T *__restrict__ v0, const T *__restrict__ v1, int64_t n, int q,
                                           const T *__restrict__ X, MulAcc<T> (&acc)[NM][BS][PW])
{
    for (int k = k0; k < k1; ++k) {
        const int col = ld_stream(scol + (b0 + k) * 32 + lane);
        T a[NM][BS * BS];
#pragma unroll
        for (int e = 0; e < BS * BS; ++e) {
            const int64_t o = ((b0 + k) * (BS * BS) + e) * 32 + lane;
            a[0][e] = __ldg(v0 + o);
            if (NM == 2) a[NM - 1][e] = __ldg(v1 + o);
        }
#pragma unroll
        for (int cc = 0; cc < BS; ++cc) {
            T xv[PW];
            ld_cols<NC>(panel_row(X, n, q, (int64_t)BS * col + cc), xv);
#pragma unroll
            for (int m = 0; m < NM; ++m)
#pragma unroll
                for (int r = 0; r < BS; ++r)
#pragma unroll
                    for (int c = 0; c < NC; ++c) acc[m][r][c].add(a[m][r * BS + cc], xv[c]);
        }
    }
}

// A's pattern with two sets of values (v1 unused without PAIR); a last panel of at
// most four columns is computed as four (its padding stays zero)
template <int BS, typename T, bool PAIR>
__global__ void __launch_bounds__(kT)
    k_spmm_parts(int64_t nb, int64_t ns, const int64_t *__restrict__ sptr, const int *__restrict__ scol,
                 const T *__restrict__ v0, const T *__restrict__ v1, int np, int cols,
                 const T *__restrict__ X, T *__restrict__ Y0, T *__restrict__ Y1, const uint8_t *__restrict__ fixed)
{
    using A = MulAcc<T>;
    constexpr int NM = PAIR ? 2 : 1, kGroups = kT / 32 / kParts<T>;
    extern __shared__ __align__(16) unsigned char smraw[];
    T *sm = reinterpret_cast<T *>(smraw);  // [group][part - 1][matrix][r][c][lane]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, grp = w / kParts<T>, part = w % kParts<T>;
    const int64_t n = nb * BS;
    for (int64_t u0 = (int64_t)blockIdx.x * kGroups; u0 < ns * np; u0 += (int64_t)gridDim.x * kGroups) {
        const int64_t u = u0 + grp;
        const bool on = u < ns * np;
        const int64_t s = on ? u / np : 0;
        const int q = on ? (int)(u - s * np) : 0;
        A acc[NM][BS][PW];
#pragma unroll
        for (int m = 0; m < NM; ++m)
#pragma unroll
            for (int r = 0; r < BS; ++r)
#pragma unroll
                for (int c = 0; c < PW; ++c) acc[m][r][c].zero();
        if (on) {
            const int64_t b0 = sptr[s];
            const int wdt = (int)(sptr[s + 1] - b0);
            const int k0 = wdt * part / kParts<T>, k1 = wdt * (part + 1) / kParts<T>;
            if (cols - q * PW > PW / 2)
                spmm_slots<BS, PW, T, NM>(b0, k0, k1, lane, scol, v0, v1, n, q, X, acc);
            else
                spmm_slots<BS, PW / 2, T, NM>(b0, k0, k1, lane, scol, v0, v1, n, q, X, acc);
        }
        T *mine = sm + (size_t)(grp * (kParts<T> - 1) + part - 1) * (NM * BS * PW * 32) + lane;
        if (part > 0)
#pragma unroll
            for (int m = 0; m < NM; ++m)
#pragma unroll
                for (int r = 0; r < BS; ++r)
#pragma unroll
                    for (int c = 0; c < PW; ++c) mine[((m * BS + r) * PW + c) * 32] = acc[m][r][c].get();
        __syncthreads();
        const int64_t row = s * 32 + lane;
        if (part == 0 && on && row < nb) {
            const T *first = sm + (size_t)grp * (kParts<T> - 1) * (NM * BS * PW * 32) + lane;
#pragma unroll
            for (int m = 0; m < NM; ++m)
#pragma unroll
                for (int r = 0; r < BS; ++r) {
                    const int64_t i = (int64_t)BS * row + r;
                    const bool f = fixed && fixed[i];
                    T yv[PW];
#pragma unroll
                    for (int c = 0; c < PW; ++c) {
                        T v = acc[m][r][c].get();
#pragma unroll
                        for (int g = 0; g < kParts<T> - 1; ++g)
                            v = A::sum(v, first[(size_t)g * (NM * BS * PW * 32) + ((m * BS + r) * PW + c) * 32]);
                        yv[c] = f ? A::none() : v;
                    }
                    st_row((m == 0 ? Y0 : Y1) + ((int64_t)q * n + i) * PW, yv);
                }
        }
        __syncthreads();
    }
}

// *same = 0 where two arrays differ
template <typename I>
__global__ void k_compare(int64_t n, const I *__restrict__ a, const I *__restrict__ b, int *same)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (a[i] != b[i]) *same = 0;
}

// k_lincomb with the blocks, the coefficients and the results in double-float.
__global__ void __launch_bounds__(kT)
    k_lincomb_df(int64_t n, int k, int nblk,
                 const __grid_constant__ CombSet<float2> set, const double *__restrict__ C)
{
    const float2 *__restrict__ X = set.X[blockIdx.y];
    const float2 *__restrict__ W = set.W[blockIdx.y];
    const float2 *__restrict__ P = set.P[blockIdx.y];
    float2 *__restrict__ Xn = set.Xn[blockIdx.y];
    float2 *__restrict__ Pn = set.Pn[blockIdx.y];
    extern __shared__ __align__(16) unsigned char smraw[];
    float2 *sC = (float2 *)smraw;
    const int m = nblk * k;
    const int np = (k + PW - 1) / PW;
    const int kp = np * PW;
    for (int e = threadIdx.x; e < m * kp; e += blockDim.x) {
        const int r = e / kp, j = e - r * kp;
        const float2 v = j < k ? df_split(C[(int64_t)j * m + r]) : make_float2(0.f, 0.f);
        float *at = reinterpret_cast<float *>(sC + (e & ~1)) + (e & 1);  // two heads, two tails
        at[0] = v.x;
        at[2] = v.y;
    }
    __syncthreads();
    for (int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < n; row += (int64_t)gridDim.x * blockDim.x) {
        for (int qo = 0; qo < np; ++qo) {
            DFRowAcc ax, ap;
            ax.zero();
            ap.zero();
            const bool half = k - qo * PW <= PW / 2;  // (the padding stays zero)
            auto block = [&](const float2 *S, int b, DFRowAcc &acc) {
                for (int qi = 0; qi < np; ++qi) {
                    float2 v[PW];
                    ld_row(panel_row(S, n, qi, row), v);
#pragma unroll
                    for (int c = 0; c < PW; ++c) {
                        const int i = qi * PW + c;
                        if (i >= k) break;
                        const float2 *at = sC + (b * k + i) * kp + qo * PW;
                        DFRow cr;
                        if (half) {
                            cr.load_paired<PW / 2>(at);
                            acc.add<PW / 2>(v[c], cr);
                        } else {
                            cr.load_paired<PW>(at);
                            acc.add<PW>(v[c], cr);
                        }
                    }
                }
            };
            block(X, 0, ax);
            for (int b = 1; b < nblk; ++b) block(b == 1 ? W : P, b, ap);
            float2 pv[PW], xv[PW];
#pragma unroll
            for (int o = 0; o < PW; ++o) {
                pv[o] = ap.get(o);
                xv[o] = df_add(ax.get(o), pv[o]);
            }
            st_row(Pn + ((int64_t)qo * n + row) * PW, pv);
            st_row(Xn + ((int64_t)qo * n + row) * PW, xv);
        }
    }
}

// Rows staged in shared memory per step.  16, 32, 48 and 64 rows took 34, 29, 27 and
// 27 us (FP32) and 90, 94, 85 and 105 us (double-float) at 70k rows and 12 columns, and
// 356, 256, 228, 210 and 1,302, 1,177, 1,167, 1,160 us at 398k and 24.
constexpr int kGramRows = 48;
constexpr int kGramSub = 4;    // each thread owns a 4 x 4 sub-tile of both Gram matrices

// Shared-memory tile of the Gram staging: kGramRows rows of one 8-column
// panel, row-major, followed by 64 bytes of padding so that consecutive tiles
// start 16 banks apart (the 16-byte loads of the threads of a quarter warp,
// which read two neighbouring tiles, then hit distinct banks).
template <typename St>
__host__ __device__ constexpr int gram_tile_elems()
{
    return kGramRows * PW + 64 / (int)sizeof(St);
}

// 16-byte moves of staged values: global (T) -> shared (St), 16 bytes of
// source per call.
__device__ __forceinline__ void gram_stage16(const float *src, float *dst)
{
    *reinterpret_cast<float4 *>(dst) = __ldg(reinterpret_cast<const float4 *>(src));
}
__device__ __forceinline__ void gram_stage16(const double *src, double *dst)
{
    *reinterpret_cast<double2 *>(dst) = __ldg(reinterpret_cast<const double2 *>(src));
}
__device__ __forceinline__ void gram_stage16(const float2 *src, float2 *dst)  // two heads, two tails
{
    const float4 w = __ldg(reinterpret_cast<const float4 *>(src));
    *reinterpret_cast<float4 *>(dst) = make_float4(w.x, w.z, w.y, w.w);
}

// A thread's 4 x 4 sums of one Gram matrix by panel type, s y^T added per row (four
// staged values each, 16-byte shared loads): FP32 panels in FP32 over the CTA's rows
// (the CTAs' sums are added in FP64), FP64 panels in FP64, double-float panels (the
// mixed mode's second phase) in double-float.
template <typename T>
struct GramTile {
    struct Four {
        T v[kGramSub];
        __device__ explicit Four(const float *p)
        {
            const float4 w = *reinterpret_cast<const float4 *>(p);
            v[0] = w.x;
            v[1] = w.y;
            v[2] = w.z;
            v[3] = w.w;
        }
        __device__ explicit Four(const double *p)
        {
            const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
            v[0] = a.x;
            v[1] = a.y;
            v[2] = b.x;
            v[3] = b.y;
        }
    };
    using Left = Four;
    using Right = Four;
    T a[kGramSub][kGramSub];
    __device__ void zero()
    {
#pragma unroll
        for (int i = 0; i < kGramSub; ++i)
#pragma unroll
            for (int j = 0; j < kGramSub; ++j) a[i][j] = T(0);
    }
    __device__ void add(int i, const Left &s, const Right &y)
    {
#pragma unroll
        for (int j = 0; j < kGramSub; ++j) a[i][j] = fma(s.v[i], y.v[j], a[i][j]);
    }
    __device__ double get(int i, int j) const { return (double)a[i][j]; }
};
template <>
struct GramTile<float2> {
    struct Left {
        float4 p[2];  // two heads, two tails
        __device__ explicit Left(const float2 *q)
        {
            p[0] = reinterpret_cast<const float4 *>(q)[0];
            p[1] = reinterpret_cast<const float4 *>(q)[1];
        }
        __device__ float2 at(int i) const
        {
            const float4 w = p[i >> 1];
            return (i & 1) ? make_float2(w.y, w.w) : make_float2(w.x, w.z);
        }
    };
    struct Right {
        ulonglong2 p[2];
        __device__ explicit Right(const float2 *q)
        {
            p[0] = reinterpret_cast<const ulonglong2 *>(q)[0];
            p[1] = reinterpret_cast<const ulonglong2 *>(q)[1];
        }
    };
    DFAcc2 a[kGramSub][2];
    __device__ void zero()
    {
#pragma unroll
        for (int i = 0; i < kGramSub; ++i) {
            a[i][0].zero();
            a[i][1].zero();
        }
    }
    __device__ void add(int i, const Left &s, const Right &y)
    {
        const DFLeft f(s.at(i));
        a[i][0].add(f, y.p[0].x, y.p[0].y);
        a[i][1].add(f, y.p[1].x, y.p[1].y);
    }
    __device__ double get(int i, int j) const { return a[i][j >> 1].get(j & 1).get(); }
};

// Upper triangles of S^T (K S) and S^T (M S), S = [X W P] (nblk blocks of k
// columns, each padded to kp = 8 np columns): each CTA reduces a contiguous
// row range and writes its partial sums (FP64) to part[cta][2 * npairs], pair
// p = (i, j), i <= j, numbered row by row over the upper triangle of the
// m = nblk k real columns.
//
// Register-tiled outer products: each block's k columns are cut into groups of
// four, and a thread takes the 4 x 4 tile of a pair of groups I <= J (G (G + 1) / 2
// threads for G = nblk ceil(k / 4) groups, at most 300; no tile below the diagonal
// and none of the padding alone: 45 threads at k = 12 where 8 x 8 tiles took 84).  A step stages kGramRows rows of every panel of S, K S and M S
// into shared memory, one panel tile after another: the rows of a panel are
// contiguous in global memory, so each warp copies whole tiles with 16-byte
// loads.  Per staged row a thread reads its 4 values of S and 4 of each image
// with 16-byte shared loads and does 32 multiply-adds: FP32 for FP32 panels
// (per CTA row range; the ranges are summed in FP64), FP64 for FP64 panels,
// or double-float (DF: double-float panels of the mixed mode's second phase)
// on the FP32 pipe.  Padding columns are staged as they are
// stored and their sums are not written.
template <typename T>
__global__ void __launch_bounds__(320)
    k_gram(int64_t n, int k, int nblk, const T *S0, const T *S1, const T *S2, const T *K0, const T *K1, const T *K2,
           const T *M0, const T *M1, const T *M2, double *part)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int kp = (k + PW - 1) / PW * PW;
    const int np = kp / PW;
    const int mp = nblk * kp;
    const int m = nblk * k;
    const int npairs = m * (m + 1) / 2;
    const int tiles = mp / PW;
    const int per_block = (k + kGramSub - 1) / kGramSub, groups = nblk * per_block;
    const int ntasks = groups * (groups + 1) / 2;
    constexpr int TE = gram_tile_elems<T>();
    T *sS = (T *)smraw;  // [3][tiles][TE]: S, K S, M S
    const bool active = (int)threadIdx.x < ntasks;
    int ti = 0, tj = 0, oi = 0, oj = 0;
    if (active) {
        int I = 0, rem = threadIdx.x;
        while (rem >= groups - I) {
            rem -= groups - I;
            ++I;
        }
        const int J = I + rem;
        const int ci = I % per_block * kGramSub, cj = J % per_block * kGramSub;  // within the blocks
        ti = I / per_block * np + ci / PW;
        tj = J / per_block * np + cj / PW;
        oi = ci % PW;
        oj = cj % PW;
    }
    GramTile<T> aA, aB;
    aA.zero();
    aB.zero();
    const int64_t per = (n + gridDim.x - 1) / gridDim.x;
    const int64_t r0 = (int64_t)blockIdx.x * per, r1 = min(n, r0 + per);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    constexpr int kPer16 = 16 / (int)sizeof(T);  // source values per 16-byte move
    const T *pS = sS + ti * TE + oi, *pK = sS + (tiles + tj) * TE + oj, *pM = sS + (2 * tiles + tj) * TE + oj;
    for (int64_t t0 = r0; t0 < r1; t0 += kGramRows) {
        const int rows = (int)((r1 - t0) < (int64_t)kGramRows ? (r1 - t0) : (int64_t)kGramRows);
        const int units = rows * PW / kPer16;  // 16-byte moves per tile
        __syncthreads();
        for (int ta = wid; ta < 3 * tiles; ta += nwarps) {
            const int mat = ta / tiles, t = ta - mat * tiles;
            const int b = t / np, q = t - b * np;
            const T *base = mat == 0 ? (b == 0 ? S0 : (b == 1 ? S1 : S2))
                                     : (mat == 1 ? (b == 0 ? K0 : (b == 1 ? K1 : K2)) : (b == 0 ? M0 : (b == 1 ? M1 : M2)));
            const T *src = base + ((int64_t)q * n + t0) * PW;
            T *dst = sS + ta * TE;
            for (int u = lane; u < units; u += 32) gram_stage16(src + u * kPer16, dst + u * kPer16);
        }
        __syncthreads();
        if (active) {
            for (int r = 0; r < rows; ++r) {
                const typename GramTile<T>::Left si(pS + r * PW);
                const typename GramTile<T>::Right yk(pK + r * PW), ym(pM + r * PW);
#pragma unroll
                for (int a = 0; a < kGramSub; ++a) {
                    aA.add(a, si, yk);
                    aB.add(a, si, ym);
                }
            }
        }
    }
    if (!active) return;
#pragma unroll
    for (int a = 0; a < kGramSub; ++a)
#pragma unroll
        for (int b = 0; b < kGramSub; ++b) {
            const int pi = PW * ti + oi + a, pj = PW * tj + oj + b;  // padded columns
            const int bi = pi / kp, ci = pi - bi * kp, bj = pj / kp, cj = pj - bj * kp;
            if (ci >= k || cj >= k) continue;
            const int i = bi * k + ci, j = bj * k + cj;
            if (i > j) continue;
            const int p = i * m - i * (i - 1) / 2 + (j - i);
            part[(int64_t)blockIdx.x * 2 * npairs + p] = aA.get(a, b);
            part[(int64_t)blockIdx.x * 2 * npairs + npairs + p] = aB.get(a, b);
        }
}

// Sum the per-CTA partials (deterministic): a CTA takes 8 values, 32 threads a share
// of the partials of each, added in thread order.  The additions alone hold the FP64
// pipe (1,520 partials of 1,332 values are 2 M, 4 us over all SMs), so the values go to
// as many SMs as there are: 15 us with 32 values to a CTA, 8 now (a thread per
// value that ran through the partials alone: 55).
constexpr int kReduceValues = 8;
__global__ void __launch_bounds__(256)
    k_reduce_parts(const double *__restrict__ part, int nparts, int len, double *__restrict__ out)
{
    __shared__ double sums[32][kReduceValues + 1];
    const int v = threadIdx.x % kReduceValues, g = threadIdx.x / kReduceValues;
    const int i = blockIdx.x * kReduceValues + v;
    double s = 0.0;
    if (i < len)
#pragma unroll 8
        for (int b = g; b < nparts; b += 32) s += part[(int64_t)b * len + i];
    sums[g][v] = s;
    __syncthreads();
    if (g == 0 && i < len) {
        double t = 0.0;
        for (int k = 0; k < 32; ++k) t += sums[k][v];
        out[i] = t;
    }
}

// The residuals' partials (per column |R|^2, |MX|^2, max|R|) of nparts CTAs: a warp
// per entry.
__global__ void k_reduce_residual(const double *__restrict__ part, int nparts, int len, double *__restrict__ out)
{
    const int lane = threadIdx.x & 31, e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (e >= len) return;
    const bool top = e % 3 == 2;
    double v = 0.0;
    for (int b = lane; b < nparts; b += 32) {
        const double x = part[(int64_t)b * len + e];
        v = top ? fmax(v, x) : v + x;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, v, o);
        v = top ? fmax(v, x) : v + x;
    }
    if (lane == 0) out[e] = v;
}

// Pn = W C_w + P C_p ; Xn = X C_x + Pn   (C: m x k column-major, FP64).
// A thread per row and output panel.  The coefficients are staged transposed,
// sC[(b k + i) kp + j] with j padded to kp by zeros, so the 8 coefficients of
// one input value for one output panel are a 16-byte-aligned row of shared
// memory (2 or 4 vector loads per 8 multiply-adds); the input and output rows
// move with 16-byte accesses.
template <typename T>
__global__ void __launch_bounds__(kT)
    k_lincomb(int64_t n, int k, int nblk, const __grid_constant__ CombSet<T> set, const double *__restrict__ C)
{
    const T *__restrict__ X = set.X[blockIdx.y];
    const T *__restrict__ W = set.W[blockIdx.y];
    const T *__restrict__ P = set.P[blockIdx.y];
    T *__restrict__ Xn = set.Xn[blockIdx.y];
    T *__restrict__ Pn = set.Pn[blockIdx.y];
    extern __shared__ __align__(16) unsigned char smraw[];
    T *sC = (T *)smraw;
    const int m = nblk * k;
    const int np = (k + PW - 1) / PW;
    const int kp = np * PW;
    for (int e = threadIdx.x; e < m * kp; e += blockDim.x) {
        const int r = e / kp, j = e - r * kp;
        sC[e] = j < k ? (T)C[(int64_t)j * m + r] : T(0);
    }
    __syncthreads();
    for (int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < n; row += (int64_t)gridDim.x * blockDim.x) {
        for (int qo = 0; qo < np; ++qo) {
            T ax[PW], ap[PW];
#pragma unroll
            for (int c = 0; c < PW; ++c) ax[c] = ap[c] = T(0);
            for (int b = 0; b < nblk; ++b) {
                for (int qi = 0; qi < np; ++qi) {
                    T v[PW];
                    ld_row(panel_row(b == 0 ? X : (b == 1 ? W : P), n, qi, row), v);
#pragma unroll
                    for (int c = 0; c < PW; ++c) {
                        const int i = qi * PW + c;
                        if (i >= k) break;
                        T cr[PW];
                        lds_row(sC + (int64_t)(b * k + i) * kp + qo * PW, cr);
#pragma unroll
                        for (int o = 0; o < PW; ++o) {
                            if (b == 0)
                                ax[o] = fma(v[c], cr[o], ax[o]);
                            else
                                ap[o] = fma(v[c], cr[o], ap[o]);
                        }
                    }
                }
            }
#pragma unroll
            for (int o = 0; o < PW; ++o) ax[o] += ap[o];
            st_row(Pn + ((int64_t)qo * n + row) * PW, ap);
            st_row(Xn + ((int64_t)qo * n + row) * PW, ax);
        }
    }
}

// R = KX - MX diag(lam); per column: |R_j|^2, |MX_j|^2, max|R_j|  -> part[cta][3k]
// (entry 3 j + {0, 1, 2} of CTA x's row).  CTA (x, q) takes the rows of panel
// q, so a thread's sums are 3 x 8 registers and its rows move as vectors.  The
// sums are FP64 (no FP32 underflow of squares for badly scaled systems); what bounds
// a small system is adding them across the CTA on the FP64 pipe, so the 16 sums
// are halved from lane to lane (16 additions per warp instead of 80) and FP32
// maxima stay FP32, and a thread takes two rows or more: 56 -> 14 us at 70k rows, k = 12.
// double-float panels: the difference on the FP32 pipe (lam split once per
// column), the sums of the leading floats (seven digits are all a norm needs).
__device__ __forceinline__ float res_lam(float, double l) { return (float)l; }
__device__ __forceinline__ double res_lam(double, double l) { return l; }
__device__ __forceinline__ float2 res_lam(float2, double l) { return df_split(-l); }
__device__ __forceinline__ float res_diff(float k, float m, float l) { return k - m * l; }
__device__ __forceinline__ double res_diff(double k, double m, double l) { return k - m * l; }
__device__ __forceinline__ float2 res_diff(float2 k, float2 m, float2 l)
{
    DFAcc a;  // k + m (-lam)
    a.hi = k.x;
    a.lo = k.y;
    a.add(m, l);
    return a.get2();
}
__device__ __forceinline__ float res_head(float v) { return v; }
__device__ __forceinline__ double res_head(double v) { return v; }
__device__ __forceinline__ float res_head(float2 v) { return v.x; }
__device__ __forceinline__ void res_zero(float &v) { v = 0.f; }
__device__ __forceinline__ void res_zero(double &v) { v = 0.0; }
__device__ __forceinline__ void res_zero(float2 &v) { v = make_float2(0.f, 0.f); }
__device__ __forceinline__ float res_max(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double res_max(double a, double b) { return fmax(a, b); }

template <typename T>
__global__ void __launch_bounds__(kT)
    k_residual(int64_t n, int k, const T *__restrict__ KX, const T *__restrict__ MX, const double *__restrict__ lam,
               T *__restrict__ R, double *part)
{
    using H = decltype(res_head(T()));  // float or double
    __shared__ double sred[2 * PW][kT / 32];
    __shared__ H smax[PW][kT / 32];
    const int q = blockIdx.y;
    double v[2 * PW];  // |R|^2 of the panel's columns, then |MX|^2
    H mx[PW];
    T lq[PW];
#pragma unroll
    for (int c = 0; c < PW; ++c) {
        v[c] = v[PW + c] = 0.0;
        mx[c] = H(0);
        lq[c] = res_lam(T(), q * PW + c < k ? lam[q * PW + c] : 0.0);
    }
    for (int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < n; row += (int64_t)gridDim.x * blockDim.x) {
        const int64_t off = ((int64_t)q * n + row) * PW;
        T kv[PW], mv[PW];
        ld_row(KX + off, kv);
        ld_row(MX + off, mv);
#pragma unroll
        for (int c = 0; c < PW; ++c) {
            if (q * PW + c >= k) {
                res_zero(kv[c]);
                continue;
            }
            kv[c] = res_diff(kv[c], mv[c], lq[c]);
            const H r = res_head(kv[c]);
            const double rd = (double)r, md = (double)res_head(mv[c]);
            v[c] = fma(rd, rd, v[c]);
            v[PW + c] = fma(md, md, v[PW + c]);
            mx[c] = res_max(mx[c], r < H(0) ? -r : r);
        }
        st_row(R + off, kv);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // lane l ends up with value l >> 1 over the warp
#pragma unroll
    for (int h = PW, o = 16; h > 0; h >>= 1, o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double send = upper ? v[i] : v[i + h];
            const double stay = upper ? v[i + h] : v[i];
            v[i] = stay + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    if ((lane & 1) == 0) sred[lane >> 1][wid] = v[0];
#pragma unroll
    for (int c = 0; c < PW; ++c) {
        H m = mx[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = res_max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) smax[c][wid] = m;
    }
    __syncthreads();
    if (threadIdx.x < 3 * PW) {
        const int c = threadIdx.x / 3, t = threadIdx.x % 3;
        if (q * PW + c < k) {
            double x = 0.0;
            for (int w = 0; w < kT / 32; ++w)
                x = t == 2 ? fmax(x, (double)smax[c][w]) : x + sred[t * PW + c][w];
            part[(int64_t)blockIdx.x * 3 * k + 3 * (q * PW + c) + t] = x;
        }
    }
}

// k_eig_precond for double-float panels, in double-float arithmetic (the
// block inverse split once per node).
template <int BS>
__global__ void __launch_bounds__(kT)
    k_eig_precond_df(int64_t nb, int k, const double *__restrict__ dinv, int pc, const float2 *__restrict__ R,
                     float2 *__restrict__ W, const uint8_t *__restrict__ fixed)
{
    const int np = (k + PW - 1) / PW;
    const int64_t n = nb * BS;
    for (int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; node < nb;
         node += (int64_t)gridDim.x * blockDim.x) {
        float2 D[BS * BS];
#pragma unroll
        for (int e = 0; e < BS * BS; ++e)
            D[e] = pc == PFG_PC_NONE ? make_float2(e % (BS + 1) == 0 ? 1.f : 0.f, 0.f)
                                     : df_split(dinv[node * BS * BS + e]);
        for (int q = 0; q < np; ++q) {
            float2 rv[BS][PW];
#pragma unroll
            for (int i = 0; i < BS; ++i) ld_row(panel_row(R, n, q, (int64_t)BS * node + i), rv[i]);
#pragma unroll
            for (int i = 0; i < BS; ++i) {
                const bool f = fixed && fixed[(int64_t)BS * node + i];
                float2 wv[PW];
#pragma unroll
                for (int c = 0; c < PW; ++c) {
                    DFAcc a;
                    a.zero();
#pragma unroll
                    for (int j = 0; j < BS; ++j) a.add(D[BS * i + j], rv[j][c]);
                    wv[c] = f ? make_float2(0.f, 0.f) : a.get2();
                }
                st_row(W + ((int64_t)q * n + (int64_t)BS * node + i) * PW, wv);
            }
        }
    }
}

// W = T R: block Jacobi (BS x BS diagonal blocks of K) per node and column;
// fixed DOFs zeroed.
template <int BS, typename T>
__global__ void __launch_bounds__(kT)
    k_eig_precond(int64_t nb, int k, const double *__restrict__ dinv, int pc, const T *__restrict__ R,
                  T *__restrict__ W, const uint8_t *__restrict__ fixed)
{
    const int np = (k + PW - 1) / PW;
    const int64_t n = nb * BS;
    for (int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; node < nb;
         node += (int64_t)gridDim.x * blockDim.x) {
        // the phase's own precision: FP32 panels take the block inverse in FP32
        using W_t = typename std::conditional<std::is_same<T, float>::value, float, double>::type;
        W_t D[BS * BS];
#pragma unroll
        for (int e = 0; e < BS * BS; ++e)
            D[e] = pc == PFG_PC_NONE ? (e % (BS + 1) == 0 ? W_t(1) : W_t(0)) : (W_t)dinv[node * BS * BS + e];
        for (int q = 0; q < np; ++q) {
            T rv[BS][PW];
#pragma unroll
            for (int i = 0; i < BS; ++i) ld_row(panel_row(R, n, q, (int64_t)BS * node + i), rv[i]);
#pragma unroll
            for (int i = 0; i < BS; ++i) {
                const bool f = fixed && fixed[(int64_t)BS * node + i];
                T wv[PW];
#pragma unroll
                for (int c = 0; c < PW; ++c) {
                    W_t v = W_t(0);
#pragma unroll
                    for (int j = 0; j < BS; ++j) v += D[BS * i + j] * (W_t)rv[j][c];
                    wv[c] = f ? T(0) : (T)v;
                }
                st_row(W + ((int64_t)q * n + (int64_t)BS * node + i) * PW, wv);
            }
        }
    }
}

__device__ __forceinline__ uint64_t splitmix(uint64_t x)
{
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// X = uniform(-1, 1) from (seed, row, column); padding columns and fixed rows 0.
template <typename T>
__global__ void k_random(int64_t n, int k, uint64_t seed, T *__restrict__ X, const uint8_t *__restrict__ fixed)
{
    const int np = (k + PW - 1) / PW;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n * np * PW;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % PW);
        const int64_t row = (i / PW) % n;
        const int q = (int)(i / (PW * n));
        const int j = q * PW + c;
        const uint64_t h = splitmix(seed * 0x100000001b3ull ^ splitmix((uint64_t)row * 131 + (uint64_t)j));
        const double u = (double)(h >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
        X[i] = (j < k && !(fixed && fixed[row])) ? (T)u : T(0);
    }
}

__device__ __forceinline__ float2 to_df32(float x) { return make_float2(x, 0.f); }
__device__ __forceinline__ double to_f64(float x) { return (double)x; }
__device__ __forceinline__ double to_f64(double x) { return x; }
__device__ __forceinline__ double to_f64(float2 x) { return df_value(x); }

// FP32 panels -> double-float panels (the start of the mixed second phase)
__global__ void k_f32_to_df(int64_t len, const float *__restrict__ a, float2 *__restrict__ b)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = to_df32(a[i]);
}

// first nev columns of X (panels) -> column-major n x nev (FP64)
template <typename T>
__global__ void k_unpanel(int64_t n, int nev, const T *__restrict__ X, double *__restrict__ out)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n * nev; i += (int64_t)gridDim.x * blockDim.x) {
        const int j = (int)(i / n);
        const int64_t row = i - (int64_t)j * n;
        out[i] = to_f64(X[((int64_t)(j / PW) * n + row) * PW + (j % PW)]);
    }
}

// ===================================================================== driver
namespace {

int g_sms = 0;
int sms()
{
    if (!g_sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_sms <= 0) g_sms = 1;
    }
    return g_sms;
}

template <typename T>
struct Blocks {
    DevBuf<T> X, W, P, KX, KW, KP, MX, MW, MP, Xn, Pn, KXn, KPn, MXn, MPn, R;
    void alloc(size_t len)
    {
        for (DevBuf<T> *b : {&X, &W, &P, &KX, &KW, &KP, &MX, &MW, &MP, &Xn, &Pn, &KXn, &KPn, &MXn, &MPn, &R})
            b->resize(len);
    }
};

struct Ctx {
    int64_t n, nb;
    int bs;
    int k, kp, np;
    cudaStream_t st;
    const uint8_t *fixed;
    DevBuf<float2> df_K, df_M;  // the sliced FP64 matrix values as double-float pairs (mixed second phase)
    const DevMatrix *dfK = nullptr, *dfM = nullptr;
    int launches = 0;
    DevBuf<double> part, C, dinv;
    const double *lam_d = nullptr;  // behind the coefficients in C
    std::vector<double> hC, hlam;
    double *pin = nullptr;     // page-locked, read and written by the device: small matrices and sums
    cudaEvent_t sums = nullptr;  // the residuals' sums have arrived
    bool one_pattern = false;  // K and M share their sliced pattern
    int ngrid;
    ~Ctx()
    {
        if (pin) {
            cudaStreamSynchronize(st);  // (kernels write there)
            cudaFreeHost(pin);
        }
        if (sums) cudaEventDestroy(sums);
    }
};

// Ctx::pin, in doubles: both Gram triangles of three blocks of at most 32 columns and
// the residuals' sums, which the kernels that form them write straight to the host (a copy of
// its own costs more than the few KB take), then the coefficients and Ritz values.
constexpr size_t kPinSums = 96 * 97, kPinCoef = kPinSums + 3 * 32, kPinDoubles = kPinCoef + 96 * 32 + 32;

template <typename T>
SellView<T> sell_of(const DevMatrix &A)
{
    if constexpr (std::is_same<T, double>::value)
        return A.sell<double>();
    else
        return A.sell<float>();
}

// A's sliced FP64 values as double-float pairs (converted once per phase).
static const float2 *df_values(Ctx &c, const DevMatrix &A)
{
    const bool isK = &A == c.dfK;
    PFG_CHECK(isK || &A == c.dfM, PFG_E_INTERNAL, "double-float values of an unexpected matrix");
    return isK ? c.df_K.p : c.df_M.p;
}

static void to_df(Ctx &c, const double *a, float2 *b, int64_t len)
{
    k_to_df<<<grid_for(len, 256, sms() * 8), 256, 0, c.st>>>(len, a, b);
    PFG_CUDA(cudaGetLastError());
    ++c.launches;
}

// Systems of few (slice, panel) units per SM share a unit among kParts<T> warps.  A
// matrix alone: whole units win from about 50 per SM on (double-float, whole against
// shared: 351 and 349 us at 54 per SM, 552 and 593 at 93, 1,078 and 1,383 at 190); the
// fused pair pays for longer (two products against the pair: 195 and 142 us at 54, 301
// and 241 at 93, 595 and 782 at 190).
static bool few_units(const Ctx &c, const DevMatrix &A, int64_t per_sm) { return A.ns * c.np < sms() * per_sm; }
constexpr int64_t kUnitsAlone = 48, kUnitsPair = 96;

// Y0 = A X (Y1 = B X too when PAIR: values v1 on A's pattern), kParts warps per unit.
template <typename T, bool PAIR>
static void spmm_parts(Ctx &c, const DevMatrix &A, const T *v0, const T *v1, const T *X, T *Y0, T *Y1)
{
    constexpr int kGroups = kT / 32 / kParts<T>;
    const size_t smem = (size_t)kGroups * (kParts<T> - 1) * (PAIR ? 2 : 1) * A.bs * PW * 32 * sizeof(T);
    const int64_t ctas = (A.ns * c.np + kGroups - 1) / kGroups;
    const int g = (int)std::min<int64_t>(ctas, (int64_t)sms() * 64);
    if (A.bs == 3) {
        PFG_CUDA(cudaFuncSetAttribute(k_spmm_parts<3, T, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_spmm_parts<3, T, PAIR><<<g, kT, smem, c.st>>>(A.nb, A.ns, A.sptr.p, A.scol.p, v0, v1, c.np, c.k, X, Y0,
                                                        Y1, c.fixed);
    } else {
        k_spmm_parts<1, T, PAIR><<<g, kT, smem, c.st>>>(A.nb, A.ns, A.sptr.p, A.scol.p, v0, v1, c.np, c.k, X, Y0,
                                                        Y1, c.fixed);
    }
    PFG_CUDA(cudaGetLastError());
    ++c.launches;
}

// Y = A X, panels in double-float, A's values as double-float pairs.
static void spmm_df(Ctx &c, const DevMatrix &A, const float2 *X, float2 *Y)
{
    if (few_units(c, A, kUnitsAlone)) {
        spmm_parts<float2, false>(c, A, df_values(c, A), nullptr, X, Y, nullptr);
        return;
    }
    const SellView<double> v = A.sell<double>();
    int per = 0;
    if (A.bs == 3)
        PFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_spmm_df<3>, kT, 0));
    else
        PFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_spmm_df<1>, kT, 0));
    const int64_t warps = A.ns * c.np;
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, (int64_t)std::max(per, 1) * sms()));
    if (A.bs == 3)
        k_spmm_df<3><<<g, kT, 0, c.st>>>(v, df_values(c, A), c.np, X, Y, c.fixed);
    else
        k_spmm_df<1><<<g, kT, 0, c.st>>>(v, df_values(c, A), c.np, X, Y, c.fixed);
    PFG_CUDA(cudaGetLastError());
    ++c.launches;
}

template <typename T>
void spmm(Ctx &c, const DevMatrix &A, const T *X, T *Y)
{
    if constexpr (std::is_same<T, float2>::value) {
        spmm_df(c, A, X, Y);
    } else {
        if constexpr (std::is_same<T, float>::value) {
            if (few_units(c, A, kUnitsAlone)) {
                spmm_parts<float, false>(c, A, A.s32.p, nullptr, X, Y, nullptr);
                return;
            }
        }
        const SellView<T> v = sell_of<T>(A);
        int per = 0;
        if (A.bs == 3)
            PFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_spmm<3, T>, kT, 0));
        else
            PFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_spmm<1, T>, kT, 0));
        const int64_t warps = A.ns * c.np;
        const int g =
            (int)std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, (int64_t)std::max(per, 1) * sms()));
        if (A.bs == 3)
            k_spmm<3, T><<<g, kT, 0, c.st>>>(v, c.np, X, Y, c.fixed);
        else
            k_spmm<1, T><<<g, kT, 0, c.st>>>(v, c.np, X, Y, c.fixed);
        PFG_CUDA(cudaGetLastError());
        ++c.launches;
    }
}

// KX = K X and MX = M X
template <typename T>
void spmm_pair(Ctx &c, const DevMatrix &K, const DevMatrix &M, const T *X, T *KX, T *MX)
{
    if constexpr (std::is_same<T, float>::value) {
        if (c.one_pattern && few_units(c, K, kUnitsPair)) {
            spmm_parts<float, true>(c, K, K.s32.p, M.s32.p, X, KX, MX);
            return;
        }
    }
    spmm<T>(c, K, X, KX);
    spmm<T>(c, M, X, MX);
}

template <typename T>
void gram(Ctx &c, int nblk, const Blocks<T> &B, std::vector<double> &GA, std::vector<double> &GB)
{
    const int m = nblk * c.k;
    const int npairs = m * (m + 1) / 2;
    const int mp = nblk * c.kp;
    const int tiles = mp / PW;
    const int groups = nblk * ((c.k + kGramSub - 1) / kGramSub);
    const int threads = (groups * (groups + 1) / 2 + 31) / 32 * 32;
    // staged tiles: 3 matrices x tiles; a double-float value is 8 bytes like a double
    const size_t smem = (size_t)3 * tiles * (kGramRows * PW + 64 / sizeof(T)) * sizeof(T);
    auto kern = k_gram<T>;
    PFG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // about 20 warps per SM: two CTAs of ten at k = 24, seven of three at k = 12 (two of
    // three left the pipes to latency: 58 us at 70k rows, now 27), a staged step each
    int occ = 0;
    PFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem));
    const int per_sm = std::max(1, std::min(std::max(2, 20 * 32 / threads), occ));
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((c.n + kGramRows - 1) / kGramRows, (int64_t)sms() * per_sm));
    c.part.ensure((size_t)g * 2 * npairs);
    kern<<<g, threads, smem, c.st>>>(c.n, c.k, nblk, B.X.p, B.W.p, B.P.p, B.KX.p, B.KW.p, B.KP.p, B.MX.p, B.MW.p,
                                     B.MP.p, c.part.p);
    k_reduce_parts<<<(2 * npairs + kReduceValues - 1) / kReduceValues, 256, 0, c.st>>>(c.part.p, g, 2 * npairs, c.pin);
    PFG_CUDA(cudaGetLastError());
    c.launches += 2;
    PFG_CUDA(cudaStreamSynchronize(c.st));
    GA.assign((size_t)m * m, 0.0);
    GB.assign((size_t)m * m, 0.0);
    int p = 0;
    for (int i = 0; i < m; ++i)
        for (int j = i; j < m; ++j, ++p) {
            GA[(size_t)j * m + i] = GA[(size_t)i * m + j] = c.pin[p];
            GB[(size_t)j * m + i] = GB[(size_t)i * m + j] = c.pin[npairs + p];
        }
}

template <typename T>
void lincomb(Ctx &c, int nblk, const CombSet<T> &set)
{
    const int m = nblk * c.k;
    const size_t smem = (size_t)m * c.kp * sizeof(T);  // (a double-float coefficient is 8 bytes too)
    const dim3 g((unsigned)grid_for(c.n, kT, sms() * 8), 3);
    if constexpr (std::is_same<T, float2>::value) {
        PFG_CUDA(cudaFuncSetAttribute(k_lincomb_df, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_lincomb_df<<<g, kT, smem, c.st>>>(c.n, c.k, nblk, set, c.C.p);
    } else {
        PFG_CUDA(cudaFuncSetAttribute(k_lincomb<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_lincomb<T><<<g, kT, smem, c.st>>>(c.n, c.k, nblk, set, c.C.p);
    }
    PFG_CUDA(cudaGetLastError());
    ++c.launches;
}

// Rayleigh-Ritz on nblk blocks: C, lam on the device; returns pairs found.
template <typename T>
int rayleigh_ritz(Ctx &c, int nblk, const Blocks<T> &B, double rank_tol)
{
    std::vector<double> GA, GB;
    gram<T>(c, nblk, B, GA, GB);
    const int m = nblk * c.k;
    c.hC.assign((size_t)m * c.k, 0.0);
    c.hlam.assign(c.k, 0.0);
    const int got = small_generalized_eig(m, GA.data(), GB.data(), c.k, rank_tol, c.hlam.data(), c.hC.data());
    if (got < c.k) return got;
    // (the copy has left this buffer before the next synchronisation that precedes its reuse)
    const size_t len = (size_t)m * c.k;
    c.C.ensure(len + c.k);
    c.lam_d = c.C.p + len;
    std::copy(c.hC.begin(), c.hC.end(), c.pin + kPinCoef);
    std::copy(c.hlam.begin(), c.hlam.end(), c.pin + kPinCoef + len);
    PFG_CUDA(cudaMemcpyAsync(c.C.p, c.pin + kPinCoef, (len + c.k) * sizeof(double), cudaMemcpyHostToDevice, c.st));
    return got;
}

template <typename T>
void apply_rr(Ctx &c, int nblk, Blocks<T> &B)
{
    lincomb<T>(c, nblk,
               CombSet<T>{{B.X.p, B.KX.p, B.MX.p},
                          {B.W.p, B.KW.p, B.MW.p},
                          {B.P.p, B.KP.p, B.MP.p},
                          {B.Xn.p, B.KXn.p, B.MXn.p},
                          {B.Pn.p, B.KPn.p, B.MPn.p}});
    std::swap(B.X, B.Xn);
    std::swap(B.P, B.Pn);
    std::swap(B.KX, B.KXn);
    std::swap(B.KP, B.KPn);
    std::swap(B.MX, B.MXn);
    std::swap(B.MP, B.MPn);
}

struct ResInfo {
    std::vector<double> rel, maxabs;
};

// R and the residuals' sums, on their way to the host
template <typename T>
void residuals(Ctx &c, Blocks<T> &B)
{
    const int g = (int)std::min<int64_t>((c.n + 2 * kT - 1) / (2 * kT), c.ngrid);
    c.part.ensure((size_t)g * 3 * c.k);
    k_residual<T><<<dim3(g, c.np), kT, 0, c.st>>>(c.n, c.k, B.KX.p, B.MX.p, c.lam_d, B.R.p, c.part.p);
    k_reduce_residual<<<(3 * c.k + 7) / 8, 256, 0, c.st>>>(c.part.p, g, 3 * c.k, c.pin + kPinSums);
    PFG_CUDA(cudaGetLastError());
    c.launches += 2;
    PFG_CUDA(cudaEventRecord(c.sums, c.st));
}

static ResInfo read_residuals(Ctx &c)
{
    PFG_CUDA(cudaEventSynchronize(c.sums));
    const double *h = c.pin + kPinSums;
    ResInfo ri;
    ri.rel.assign(c.k, 0.0);
    ri.maxabs.assign(c.k, 0.0);
    for (int j = 0; j < c.k; ++j) {
        const double rr = h[3 * j], mm = h[3 * j + 1], mx = h[3 * j + 2];
        const double den = std::fabs(c.hlam[j]) * std::sqrt(mm);
        ri.rel[j] = den > 0 ? std::sqrt(rr) / den : std::sqrt(rr);
        ri.maxabs[j] = mx;
    }
    return ri;
}

constexpr int kRefreshImages = 10;
constexpr int kFp32Stall = 50;

// W = T R
template <typename T>
void precondition(Ctx &c, const EigConfig &cfg, Blocks<T> &B)
{
    const int gp = grid_for(c.nb, kT, sms() * 8);
    if constexpr (std::is_same<T, float2>::value) {
        if (c.bs == 3)
            k_eig_precond_df<3><<<gp, kT, 0, c.st>>>(c.nb, c.k, c.dinv.p, cfg.precond, B.R.p, B.W.p, c.fixed);
        else
            k_eig_precond_df<1><<<gp, kT, 0, c.st>>>(c.nb, c.k, c.dinv.p, cfg.precond, B.R.p, B.W.p, c.fixed);
    } else {
        if (c.bs == 3)
            k_eig_precond<3, T><<<gp, kT, 0, c.st>>>(c.nb, c.k, c.dinv.p, cfg.precond, B.R.p, B.W.p, c.fixed);
        else
            k_eig_precond<1, T><<<gp, kT, 0, c.st>>>(c.nb, c.k, c.dinv.p, cfg.precond, B.R.p, B.W.p, c.fixed);
    }
    PFG_CUDA(cudaGetLastError());
    ++c.launches;
}

// One precision phase.  start: 0 random, 1 X already holds a start block.
template <typename T>
int phase(Ctx &c, DevMatrix &K, DevMatrix &M, Blocks<T> &B, const EigConfig &cfg, bool fp32_phase, int start,
          int &iters_left, int &iters_done, double &max_rel, double &ref_r1)
{
    const size_t len = (size_t)c.n * c.kp;
    if constexpr (!std::is_same<T, float2>::value) {
        if (start == 0) {
            k_random<T><<<grid_for((int64_t)len, 256, sms() * 8), 256, 0, c.st>>>(c.n, c.k, cfg.seed, B.X.p,
                                                                                 c.fixed);
            PFG_CUDA(cudaGetLastError());
            ++c.launches;
        }
    }
    const double rank_tol = fp32_phase ? 1e-9 : 1e-13;
    spmm_pair<T>(c, K, M, B.X.p, B.KX.p, B.MX.p);
    // Rayleigh-Ritz on X alone (X of LOBPCG_CRS, SparseClass.f90:2063-2067)
    if (rayleigh_ritz<T>(c, 1, B, rank_tol) < c.k) throw Error(PFG_E_BREAKDOWN, "LOBPCG: start block is rank deficient");
    apply_rr<T>(c, 1, B);
    bool haveP = false;
    double best = 1e300, best_lsum = 1e300;
    int since_best = 0, since_refresh = 0;
    for (;;) {
        // W = T R and its images go to the stream before the residuals are read: the host's
        // tests cost no gap on the device (after the last iteration W is left over)
        residuals<T>(c, B);
        if (iters_left > 0) {
            precondition<T>(c, cfg, B);
            spmm_pair<T>(c, K, M, B.W.p, B.KW.p, B.MW.p);
        }
        const ResInfo ri = read_residuals(c);
        max_rel = 0.0;
        double maxabs = 0.0;
        for (int j = 0; j < cfg.nev; ++j) {
            max_rel = std::max(max_rel, ri.rel[j]);
            maxabs = std::max(maxabs, ri.maxabs[j]);
        }
        if (ref_r1 < 0) ref_r1 = maxabs;
        if (cfg.debug)
            fprintf(stderr, "[pfg] LOBPCG %s it %d max rel residual %.3e lambda_1 %.9e\n", fp32_phase ? "fp32" : "fp64",
                    iters_done, max_rel, c.hlam[0]);
        const bool conv = cfg.stop_rule == 0 ? (maxabs / (ref_r1 > 0 ? ref_r1 : 1.0) < cfg.tol) : (max_rel < cfg.tol);
        if (conv) return 1;
        if (fp32_phase) {
            if (max_rel < cfg.tol_fp32) return 0;
            // FP32 floor: neither the mean log residual of the wanted pairs
            // (by 10 %) nor the sum of their Ritz values (by more than FP32
            // noise, 1e-6 relative) fell for kFp32Stall iterations.  From a
            // random start the Ritz values fall for many iterations while the
            // relative residuals grow, so the residuals alone are no signal.
            double mlog = 0.0, lsum = 0.0;
            for (int j = 0; j < cfg.nev; ++j) {
                mlog += std::log(std::max(ri.rel[j], 1e-300));
                lsum += c.hlam[j];
            }
            mlog /= cfg.nev;
            const bool res_down = mlog < best - std::log(1.1);
            const bool lam_down = lsum < best_lsum - 1e-6 * std::fabs(best_lsum);
            if (res_down) best = mlog;
            if (lam_down) best_lsum = lsum;
            if (res_down || lam_down) {
                since_best = 0;
            } else if (++since_best > kFp32Stall) {
                return 0;
            }
        }
        if (iters_left <= 0) return -1;
        --iters_left;
        ++iters_done;
        int nblk = haveP ? 3 : 2;
        int got = rayleigh_ritz<T>(c, nblk, B, rank_tol);
        if (got < c.k && nblk == 3) {
            nblk = 2;  // P became dependent: drop it this iteration
            got = rayleigh_ritz<T>(c, nblk, B, rank_tol);
        }
        if (got < c.k) throw Error(PFG_E_BREAKDOWN, "LOBPCG: Rayleigh-Ritz basis lost rank");
        apply_rr<T>(c, nblk, B);
        haveP = true;
        // The images KX, MX, KP, MP follow X and P through the same linear
        // combinations; recompute them from X and P every kRefreshImages
        // iterations so rounding in those updates cannot drift the residuals
        // R = KX - MX Lambda away from the true ones (without this the FP64
        // phase stalled near 3e-3 on the 60^3 cantilever).
        if (++since_refresh >= kRefreshImages) {
            since_refresh = 0;
            spmm_pair<T>(c, K, M, B.X.p, B.KX.p, B.MX.p);
            spmm_pair<T>(c, K, M, B.P.p, B.KP.p, B.MP.p);
        }
    }
}

}  // namespace

// Block Jacobi (3x3 node blocks) inverse of K, FP64, for the LOBPCG preconditioner.
void block_jacobi_inverse(const DevMatrix &A, int pc, double *d64, cudaStream_t st);

EigResult lobpcg_solve(DevMatrix &K, DevMatrix &M, const uint8_t *fixed, const EigConfig &cfg_in, double *lambda,
                       double *Xout, cudaStream_t st)
{
    EigConfig cfg = cfg_in;
    PFG_CHECK(K.bs == M.bs && K.nb == M.nb, PFG_E_ARG, "eig: A and B must have the same size and block structure");
    if (cfg.block < cfg.nev) cfg.block = cfg.nev;
    PFG_CHECK(cfg.nev >= 1 && cfg.block <= 32, PFG_E_ARG, "eig: need 1 <= num_eigen <= block size <= 32");
    Ctx c;
    c.n = K.ndof();
    c.nb = K.nb;
    c.bs = K.bs;
    c.k = cfg.block;
    c.kp = (c.k + PW - 1) / PW * PW;
    c.np = c.kp / PW;
    c.st = st;
    c.fixed = fixed;
    c.ngrid = sms() * 2;
    PFG_CHECK(c.n >= 3 * c.k, PFG_E_ARG, "eig: block size too large for the system");
    PFG_CUDA(cudaMallocHost((void **)&c.pin, kPinDoubles * sizeof(double)));
    PFG_CUDA(cudaEventCreateWithFlags(&c.sums, cudaEventDisableTiming));
    EigResult res;
    cudaEvent_t e0, e1;
    PFG_CUDA(cudaEventCreate(&e0));
    PFG_CUDA(cudaEventCreate(&e1));
    PFG_CUDA(cudaEventRecord(e0, st));
    c.dinv.ensure((size_t)c.nb * c.bs * c.bs);
    block_jacobi_inverse(K, cfg.precond == PFG_PC_NONE ? PFG_PC_BLOCK_JACOBI : cfg.precond, c.dinv.p, st);
    ++c.launches;
    const size_t len = (size_t)c.n * c.kp;
    int iters_left = cfg.max_itr, iters_done = 0, rc = -1;
    double max_rel = 0.0, ref_r1 = -1.0;
    build_sell(K, true, cfg.precision == PFG_PREC_MIXED, st);
    build_sell(M, true, cfg.precision == PFG_PREC_MIXED, st);
    if (cfg.precision == PFG_PREC_MIXED && K.ns == M.ns && K.scol.n == M.scol.n) {
        DevBuf<int> same(1);
        int one = 1;
        PFG_CUDA(cudaMemcpyAsync(same.p, &one, sizeof(int), cudaMemcpyHostToDevice, st));
        k_compare<<<grid_for(K.ns + 1, 256), 256, 0, st>>>(K.ns + 1, K.sptr.p, M.sptr.p, same.p);
        k_compare<<<grid_for((int64_t)K.scol.n, 256), 256, 0, st>>>((int64_t)K.scol.n, K.scol.p, M.scol.p, same.p);
        PFG_CUDA(cudaGetLastError());
        PFG_CUDA(cudaMemcpyAsync(&one, same.p, sizeof(int), cudaMemcpyDeviceToHost, st));
        PFG_CUDA(cudaStreamSynchronize(st));
        c.one_pattern = one != 0;
    }
    Blocks<double> B64;
    Blocks<float2> Bdf;
    if (cfg.precision == PFG_PREC_MIXED) {
        // FP32 phase, then the second phase with the panels, images, SpMM,
        // Gram and linear combinations in double-float on the FP32 pipe (the
        // matrices' FP64 values split once here)
        {
            Blocks<float> B32;
            B32.alloc(len);
            double r1 = -1.0;
            rc = phase<float>(c, K, M, B32, cfg, true, 0, iters_left, iters_done, max_rel, r1);
            res.iterations_fp32 = iters_done;
            Bdf.alloc(len);
            k_f32_to_df<<<grid_for((int64_t)len, 256, sms() * 8), 256, 0, st>>>((int64_t)len, B32.X.p, Bdf.X.p);
            PFG_CUDA(cudaGetLastError());
            ++c.launches;
        }
        c.dfK = &K;
        c.dfM = &M;
        c.df_K.resize(K.s64.n);
        c.df_M.resize(M.s64.n);
        to_df(c, K.s64.p, c.df_K.p, (int64_t)K.s64.n);
        to_df(c, M.s64.p, c.df_M.p, (int64_t)M.s64.n);
        rc = phase<float2>(c, K, M, Bdf, cfg, false, 1, iters_left, iters_done, max_rel, ref_r1);
    } else {
        B64.alloc(len);
        rc = phase<double>(c, K, M, B64, cfg, false, 0, iters_left, iters_done, max_rel, ref_r1);
    }
    res.iterations = iters_done;
    res.max_rel_residual = max_rel;
    res.status = rc == 1 ? PFG_OK : PFG_W_NOT_CONVERGED;
    for (int j = 0; j < cfg.nev; ++j) lambda[j] = c.hlam[j];
    if (Xout) {
        if (cfg.precision == PFG_PREC_MIXED)
            k_unpanel<float2><<<grid_for(c.n * cfg.nev, 256, sms() * 8), 256, 0, st>>>(c.n, cfg.nev, Bdf.X.p, Xout);
        else
            k_unpanel<double><<<grid_for(c.n * cfg.nev, 256, sms() * 8), 256, 0, st>>>(c.n, cfg.nev, B64.X.p, Xout);
        PFG_CUDA(cudaGetLastError());
        ++c.launches;
    }
    PFG_CUDA(cudaEventRecord(e1, st));
    PFG_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    res.ms = ms;
    res.launches = c.launches;
    return res;
}

}  // namespace pfg
