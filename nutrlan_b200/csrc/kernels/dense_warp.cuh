// Warp-parallel forms of the small dense routines the batched solver runs at
// every restart (host/dense_core.h): implicit QL with eigenvector
// accumulation, Householder tridiagonalisation with Q, the symmetric
// eigen-solve built on them, and trl_get_eval / trl_get_tvec /
// trl_get_tvec_a / trl_tridiag.  All 32 lanes of one warp call them with
// their lane index.  The algorithms are those of the serial code:
//   * QL: every lane runs the scalar bulge chase on the shared d and e (lane
//     0 writes them) and applies the plane rotations to its own rows of Z
//     (rows k = lane, lane + 32, ...).  The chase is one dependent chain, so
//     it decides the time: a rotation takes one reciprocal square root and a
//     correction instead of hypot and two divisions, its inputs are loaded
//     one rotation ahead, the column shared by two rotations stays in a
//     register, and the negligible off-diagonal is found by all lanes.  The
//     lanes meet after every rotation;
//   * Householder: p = tau A v by rows, the rank-2 update by columns, Q by
//     columns; the reflector scalars are computed redundantly.
// Shared arrays written by one lane and read by others are separated by
// __syncwarp().
#pragma once

#include <cfloat>

#include "../host/dense_core.h"

namespace trlb {
namespace warp {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxN = 66;  // largest projected problem (maxlan + 2)

// (c, s) = (g, f) / r with r = |(f, g)|; false when r is zero.
__device__ __forceinline__ bool rotation(double f, double g, double &r, double &s, double &c) {
    const double r2 = fma(f, f, g * g);
    if (r2 > 1e-280 && r2 < 1e280) {
        const double ir = rsqrt(r2);
        r = r2 * ir;
        s = f * ir;
        c = g * ir;
        // s^2 + c^2 is 1 to a few roundings: one step towards 1.
        const double t = 0.5 * fma(-s, s, fma(-c, c, 1.0));
        s = fma(t, s, s);
        c = fma(t, c, c);
        return true;
    }
    r = hypot(f, g);
    if (r == 0.0) return false;
    s = f / r;
    c = g / r;
    return true;
}

__device__ inline int tql_implicit(int n, double *d, double *e, double *Z, int ldz, int zrows, int lane) {
    if (n <= 1) return 0;
    constexpr int RZ = (kMaxN + 31) / 32;  // rows of Z per lane
    if (lane == 0) e[n - 1] = 0.0;
    __syncwarp();
    const int max_sweeps = 60;
    for (int l = 0; l < n; ++l) {
        int sweeps = 0;
        for (;;) {
            int m = n - 1;
            for (int b = l; b < n - 1; b += 32) {
                const int q = b + lane;
                const bool tiny = q < n - 1 && fabs(e[q]) <= DBL_EPSILON * (fabs(d[q]) + fabs(d[q + 1]));
                const unsigned found = __ballot_sync(kFull, tiny);
                if (found) {
                    m = b + __ffs(found) - 1;
                    break;
                }
            }
            if (m == l) break;
            if (++sweeps > max_sweeps) return l + 1;
            double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
            double r = hypot(g, 1.0);
            g = d[m] - d[l] + e[l] / (g + (g >= 0.0 ? r : -r));
            double s = 1.0, c = 1.0, p = 0.0;
            double ei = e[m - 1], di = d[m - 1], d1 = d[m];
            double zt[RZ];  // this lane's rows of column i + 1
#pragma unroll
            for (int u = 0; u < RZ; ++u) {
                const int k = lane + 32 * u;
                zt[u] = k < zrows ? Z[(size_t)m * ldz + k] : 0.0;
            }
            __syncwarp();  // the chase below rewrites what was read here
            bool deflated = false;
            int i = m - 1;
            for (; i >= l; --i) {
                const double en = i > l ? e[i - 1] : 0.0, dn = i > l ? d[i - 1] : 0.0;
                const double f = s * ei, b = c * ei;
                const bool fine = rotation(f, g, r, s, c);
                if (lane == 0) e[i + 1] = r;
                if (!fine) {
                    deflated = true;
                    break;
                }
                g = d1 - p;
                r = (di - g) * s + 2.0 * c * b;
                p = s * r;
                if (lane == 0) d[i + 1] = g + p;
                g = c * r - b;
#pragma unroll
                for (int u = 0; u < RZ; ++u) {
                    const int k = lane + 32 * u;
                    if (k < zrows) {
                        const double zi = Z[(size_t)i * ldz + k];
                        Z[(size_t)(i + 1) * ldz + k] = s * zi + c * zt[u];
                        zt[u] = c * zi - s * zt[u];
                    }
                }
                d1 = di;
                di = dn;
                ei = en;
                // Lane 0 writes entry i + 1 of d and e and the others read
                // entry i - 1: a lane behind by two rotations would read a
                // new value.
                __syncwarp();
            }
#pragma unroll
            for (int u = 0; u < RZ; ++u) {
                const int k = lane + 32 * u;
                if (k < zrows) Z[(size_t)(i + 1) * ldz + k] = zt[u];
            }
            if (lane == 0) {
                if (deflated) {
                    d[i + 1] -= p;
                } else {
                    d[l] -= p;
                    e[l] = g;
                }
                e[m] = 0.0;
            }
            __syncwarp();
        }
    }
    return 0;
}

__device__ inline void tridiag_upper(int n, double *A, int lda, double *d, double *e, bool want_q, double *ws,
                                     int lane) {
    auto a = [&](int i, int j) -> double & { return A[(size_t)j * lda + i]; };
    if (n <= 0) return;
    double *vs = ws, *taus = ws + (size_t)n * n, *p = taus + n, *w = p + n;
    for (size_t q = lane; q < (size_t)n * n; q += 32) vs[q] = 0.0;
    for (int q = lane; q < n; q += 32) taus[q] = 0.0;
    __syncwarp();
    for (int k = n - 1; k >= 2; --k) {
        const double alpha = a(k - 1, k);
        double sigma = 0.0;
        for (int i = 0; i < k - 1; ++i) sigma += a(i, k) * a(i, k);
        double *v = &vs[(size_t)k * n];
        if (sigma == 0.0) {
            __syncwarp();
            if (lane == 0) {
                taus[k] = 0.0;
                e[k - 1] = alpha;
            }
            __syncwarp();
            continue;
        }
        const double mu = sqrt(alpha * alpha + sigma);
        const double beta = alpha <= 0.0 ? mu : -mu;
        const double tau = (beta - alpha) / beta;
        const double scal = 1.0 / (alpha - beta);
        for (int i = lane; i < k - 1; i += 32) v[i] = a(i, k) * scal;
        if (lane == 0) {
            v[k - 1] = 1.0;
            taus[k] = tau;
            e[k - 1] = beta;
        }
        __syncwarp();
        for (int i = lane; i < k; i += 32) {
            double s = 0.0;
            for (int j = 0; j < k; ++j) s += a(i, j) * v[j];
            p[i] = tau * s;
        }
        __syncwarp();
        double pv = 0.0;
        for (int i = 0; i < k; ++i) pv += p[i] * v[i];
        for (int i = lane; i < k; i += 32) w[i] = p[i] - 0.5 * tau * pv * v[i];
        __syncwarp();
        for (int j = lane; j < k; j += 32)
            for (int i = 0; i < k; ++i) a(i, j) -= v[i] * w[j] + w[i] * v[j];
        __syncwarp();
        for (int i = lane; i < k - 1; i += 32) {
            a(i, k) = 0.0;
            a(k, i) = 0.0;
        }
        if (lane == 0) {
            a(k - 1, k) = beta;
            a(k, k - 1) = beta;
        }
        __syncwarp();
    }
    if (lane == 0) {
        if (n >= 2) e[0] = a(0, 1);
        for (int i = 0; i < n; ++i) d[i] = a(i, i);
    }
    __syncwarp();
    if (!want_q) return;
    for (int j = lane; j < n; j += 32)
        for (int i = 0; i < n; ++i) a(i, j) = (i == j) ? 1.0 : 0.0;
    __syncwarp();
    for (int k = 2; k <= n - 1; ++k) {
        const double tau = taus[k];
        if (tau == 0.0) continue;
        const double *v = &vs[(size_t)k * n];
        for (int j = lane; j < n; j += 32) {
            double s = 0.0;
            for (int i = 0; i < k; ++i) s += v[i] * a(i, j);
            s *= tau;
            for (int i = 0; i < k; ++i) a(i, j) -= s * v[i];
        }
    }
    __syncwarp();
}

__device__ inline int sym_eig(int n, double *A, int lda, double *w, double *ws, int lane) {
    if (n <= 0) return 0;
    double *e = ws;
    for (int i = lane; i < n; i += 32) e[i] = 0.0;
    __syncwarp();
    tridiag_upper(n, A, lda, w, e, true, ws + n, lane);
    const int err = tql_implicit(n, w, e, A, lda, n, lane);
    if (err) return err;
    for (int i = 0; i < n - 1; ++i) {
        int k = i;
        for (int j = i + 1; j < n; ++j)
            if (w[j] < w[k]) k = j;
        __syncwarp();
        if (k != i) {
            double *ci = A + (size_t)i * lda, *ck = A + (size_t)k * lda;
            for (int r = lane; r < n; r += 32) core::hswap(ci[r], ck[r]);
            if (lane == 0) core::hswap(w[i], w[k]);
        }
        __syncwarp();
    }
    return 0;
}

__device__ inline int arrow_to_tridiag(int nd, const double *alpha, const double *beta, double *rot, double *alfrot,
                                       double *betrot, double *ws, int lane) {
    if (nd == 0) return 0;
    if (nd == 1) {
        if (lane == 0) {
            rot[0] = 1.0;
            alfrot[0] = alpha[0];
            betrot[0] = beta[0];
        }
        __syncwarp();
        return 0;
    }
    for (size_t q = lane; q < (size_t)nd * nd; q += 32) rot[q] = 0.0;
    __syncwarp();
    for (int i = lane; i < nd; i += 32) rot[(size_t)i * nd + i] = alpha[i];
    for (int i = lane; i < nd - 1; i += 32) {
        rot[(size_t)(nd - 1) * nd + i] = beta[i];
        rot[(size_t)i * nd + (nd - 1)] = beta[i];
    }
    __syncwarp();
    tridiag_upper(nd, rot, nd, alfrot, betrot, true, ws, lane);
    if (lane == 0) betrot[nd - 1] = beta[nd - 1];
    __syncwarp();
    return 0;
}

// core::match_values without a tolerance: every wanted value takes the
// nearest computed one not yet taken (the first of equals).
__device__ inline void match_nearest(int n, const double *w, int nlam, const double *lam, int *idx, int lane) {
    constexpr int R = (kMaxN + 31) / 32;
    unsigned used = 0;  // of this lane's values lane + 32 u
    for (int i = 0; i < nlam; ++i) {
        double bd = 0.0;
        int best = n;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int j = lane + 32 * u;
            if (j < n && !(used >> u & 1)) {
                const double dd = fabs(w[j] - lam[i]);
                if (best == n || dd < bd) {
                    best = j;
                    bd = dd;
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double od = __shfl_xor_sync(kFull, bd, o);
            const int ob = __shfl_xor_sync(kFull, best, o);
            if (ob < n && (best == n || od < bd || (od == bd && ob < best))) {
                best = ob;
                bd = od;
            }
        }
        if (best < n && (best & 31) == lane) used |= 1u << (best >> 5);
        if (lane == 0) idx[i] = best < n ? best : 0;  // (no value left only if one is not a number)
    }
    __syncwarp();
}

// Eigen-solve of the tridiagonal (alpha, beta) of size nd: eigenvalues
// (unordered) in ws[0 .. nd), their vectors in the columns of
// ws[2 nd .. 2 nd + nd^2).
__device__ inline int tridiag_eig(int nd, const double *alpha, const double *beta, double *ws, int lane) {
    double *d = ws, *e = ws + nd, *Z = e + nd;
    for (int i = lane; i < nd; i += 32) {
        d[i] = alpha[i];
        e[i] = (i + 1 < nd) ? beta[i] : 0.0;
    }
    for (size_t q = lane; q < (size_t)nd * nd; q += 32) Z[q] = 0.0;
    __syncwarp();
    for (int i = lane; i < nd; i += 32) Z[(size_t)i * nd + i] = 1.0;
    __syncwarp();
    return tql_implicit(nd, d, e, Z, nd, nd, lane);
}

// trl_get_eval; with `vectors` the eigenvectors stay in ws (tridiag_eig) for
// tvec_from, else only their last components are formed.
__device__ inline int get_eval(int nd, int locked, const double *alpha, const double *beta, double *lambda,
                               double *res, bool vectors, double *ws, int lane) {
    const int m = nd - locked;
    double *d = ws, *e = ws + m, *Z = e + m;
    if (vectors) {
        if (tridiag_eig(m, alpha + locked, beta + locked, ws, lane)) return -122;
    } else {
        for (int i = lane; i < m; i += 32) {
            d[i] = alpha[locked + i];
            e[i] = (i + 1 < m) ? beta[locked + i] : 0.0;
            Z[i] = i == m - 1 ? 1.0 : 0.0;
        }
        __syncwarp();
        if (tql_implicit(m, d, e, Z, 1, 1, lane)) return -122;
    }
    for (int i = lane; i < nd; i += 32) {
        lambda[i] = i < locked ? alpha[i] : d[i - locked];
        res[i] = i < locked ? 0.0 : (vectors ? Z[(size_t)(i - locked) * m + m - 1] : Z[i - locked]);
    }
    __syncwarp();
    if (lane == 0) core::sort2(m, lambda + locked, res + locked);
    __syncwarp();
    for (int i = locked + lane; i < nd; i += 32) res[i] = beta[nd - 1] * fabs(res[i]);
    __syncwarp();
    return 0;
}

// The eigenvectors of the wanted values lambda from a tridiag_eig in ws, back
// in the basis before the arrow-to-tridiagonal rotation rot (nrot columns
// from irot on).
__device__ inline void tvec_from(int nd, int irot, int nrot, const double *rot, int nlam, const double *lambda,
                                 double *yy, double *ws, int lane) {
    double *d = ws, *Z = ws + 2 * nd, *tmp = Z + (size_t)nd * nd;
    int *idx = reinterpret_cast<int *>(tmp + nd);
    match_nearest(nd, d, nlam, lambda, idx, lane);
    for (int i = 0; i < nlam; ++i)
        for (int r = lane; r < nd; r += 32) yy[(size_t)i * nd + r] = Z[(size_t)idx[i] * nd + r];
    __syncwarp();
    if (nrot > 1) {
        for (int c = 0; c < nlam; ++c) {
            double *col = yy + (size_t)c * nd + irot;
            for (int i = lane; i < nrot; i += 32) {
                double s = 0.0;
                for (int k = 0; k < nrot; ++k) s += rot[(size_t)k * nrot + i] * col[k];
                tmp[i] = s;
            }
            __syncwarp();
            for (int i = lane; i < nrot; i += 32) col[i] = tmp[i];
            __syncwarp();
        }
    }
}

__device__ inline int get_tvec(int nd, const double *alpha, const double *beta, int irot, int nrot,
                               const double *rot, int nlam, const double *lambda, double *yy, double *ws, int lane) {
    if (nlam <= 0) return 0;
    if (tridiag_eig(nd, alpha, beta, ws, lane)) return -132;
    tvec_from(nd, irot, nrot, rot, nlam, lambda, yy, ws, lane);
    return 0;
}

__device__ inline int get_tvec_a(int nd, int kept, double *alpha, const double *beta, int nlam,
                                 const double *lambda, double *yy, double *ws, int lane) {
    if (nlam <= 0) return 0;
    double *H = ws, *w = H + (size_t)nd * nd, *wsel = w + nd, *wse = wsel + nd;
    int *idx = reinterpret_cast<int *>(wse + (size_t)nd * nd + 4 * nd);
    char *used = reinterpret_cast<char *>(idx + nd);
    for (size_t q = lane; q < (size_t)nd * nd; q += 32) H[q] = 0.0;
    __syncwarp();
    for (int i = lane; i < nd; i += 32) H[(size_t)i * nd + i] = alpha[i];
    for (int i = lane; i < kept; i += 32) {
        H[(size_t)kept * nd + i] = beta[i];
        H[(size_t)i * nd + kept] = beta[i];
    }
    for (int i = kept + lane; i < nd - 1; i += 32) {
        H[(size_t)(i + 1) * nd + i] = beta[i];
        H[(size_t)i * nd + i + 1] = beta[i];
    }
    __syncwarp();
    if (sym_eig(nd, H, nd, w, wse, lane)) return -142;
    for (int i = lane; i < nd; i += 32) alpha[i] = w[i];
    __syncwarp();
    if (nlam >= nd) {
        for (size_t q = lane; q < (size_t)nd * nd; q += 32) yy[q] = H[q];
        __syncwarp();
        return 0;
    }
    const double tol = core::hmax(DBL_EPSILON * nd *
                                      core::hmax(w[nd - 1] - w[0], core::hmax(fabs(w[nd - 1]), fabs(w[0]))),
                                  DBL_MIN);
    int rc = 0;
    if (lane == 0)
        rc = core::match_values(nd, w, nlam, lambda, core::hmax(tol, core::match_tol(nd, w)), idx, used);
    rc = __shfl_sync(kFull, rc, 0);
    __syncwarp();
    if (rc != 0) return -143;
    for (int i = 0; i < nlam; ++i) {
        for (int r = lane; r < nd; r += 32) yy[(size_t)i * nd + r] = H[(size_t)idx[i] * nd + r];
    }
    if (lane == 0)
        for (int i = 0; i < nlam; ++i) wsel[i] = w[idx[i]];
    __syncwarp();
    for (int i = lane; i < nlam; i += 32) alpha[i] = wsel[i];
    __syncwarp();
    return 0;
}

}  // namespace warp
}  // namespace trlb
