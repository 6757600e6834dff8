// One cooperative kernel for a run of Lanczos steps on short vectors
// (built-in operator, FP64 / complex128 basis).
//
// Below about 10^5 rows a step is bound by latency: of launches, of grid-wide
// barriers and of the dependent loads between them.  Each block owns a
// contiguous chunk of rows for the whole run, with its rows of the basis and
// its operator entries in shared memory as far as they fit, and a step has
// one grid-wide barrier.  It is the single-sweep step of sweep.cu (the update
// of one vector and the projection of the next in one pass, the product
// corrected with A V = V T + beta q e^T), with alpha taken from the
// projection itself so that no reduction stands between the product and the
// pass:
//
//   q_k = (x - V h) / beta,  z = A q_k - beta q_{k-1} - sigma q_k
//   p = [V q_k]^H z,  g = [V q_k]^H q_k          (one reduction)
//   delta = Re p_k / g_k,  alpha = sigma + delta,  x' = z - delta q_k
//   h' = p - delta g,  |x'|^2 = |z|^2 - 2 delta Re p_k + delta^2 g_k
//
// sigma is the previous alpha.  The three sums of |x'|^2 cancel where |delta|
// is large against |x'|, so they are carried in two doubles each (compensated
// dot products: Ogita, Rump, Oishi 2005); a step with |delta| > 16 |x'| is
// logged as failed (the host takes it again with the sequential kernels).
// x' is formed by each reader from z and q_k, which every block writes to
// global memory before the barrier.  The partial sums meet in two levels: the
// blocks of a cluster through distributed shared memory, and after the grid
// barrier (one arrival per cluster) every block adds the clusters' sums itself,
// all in a fixed order.  Vectors written by other blocks are read through L2
// (ld.global.cg).  The per-step log is the one the host replays to accept or
// discard steps.
//
// A row of the operator has as many lanes as the average row needs, a long
// row a warp.  Every entry gathers from two vectors, so operators with many
// entries are better off with sweeps (coop_pays in coop.h).
//
// Measured (one B200), per step, against a kernel of five grid-wide barriers
// that read the basis twice: 128^2 lattice, basis 64, 27 -> 8 us; 12^3
// lattice, basis 40, 22 -> 8 us; complex 256^2, 37 -> 18 us; and against four
// launches a step: SELL form at 256^2, basis 48, 36 -> 11.5 us.  A step is
// three trips to L2 (the gather, the partial sums, the barrier, 1.2-1.5 us
// each) and two passes over the chunk in shared memory.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <mutex>

#include "coop.h"
#include "spmv.h"

namespace trlb {

namespace {

// 16 warps on the rows of the product and two that form the pass's
// coefficients and scalars meanwhile; all 18 in the other phases.
constexpr int kThreads = 576;

__device__ __forceinline__ double mulx(double a, double x) { return a * x; }
__device__ __forceinline__ zd mulx(zd a, zd x) { return zd{a.x * x.x - a.y * x.y, a.x * x.y + a.y * x.x}; }
__device__ __forceinline__ double shfl_x(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ zd shfl_x(zd v, int o) {
    return zd{__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o)};
}
__device__ __forceinline__ double as_c(double v, double) { return v; }
__device__ __forceinline__ zd as_c(double v, zd) { return zd{v, 0.0}; }
// acc += v * h
__device__ __forceinline__ void fma_c(double &acc, double v, double h) { acc = fma(v, h, acc); }
__device__ __forceinline__ void fma_c(zd &acc, zd v, zd h) {
    acc.x = fma(v.x, h.x, fma(-v.y, h.y, acc.x));
    acc.y = fma(v.x, h.y, fma(v.y, h.x, acc.y));
}

template <class C>
__host__ __device__ constexpr int cwidth() {
    return (int)(sizeof(C) / sizeof(double));
}
// Partial sums of a step that makes column k: p and g of columns 0 .. k, then
// |z|^2, Re p_k and g_k in two doubles each.
template <class C>
__host__ __device__ constexpr int step_doubles(int k) {
    return 2 * cwidth<C>() * (k + 1) + 6;
}

// Sum in two doubles: the value is s + c.
struct Sum2 {
    double s = 0.0, c = 0.0;
    __device__ __forceinline__ void add(double v, double e) {
        const double t = s + v, b = t - s;
        c += ((s - (t - b)) + (v - b)) + e;
        s = t;
    }
    __device__ __forceinline__ void fma2(double a, double b) {
        const double v = a * b;
        add(v, fma(a, b, -v));
    }
};
__device__ __forceinline__ void dot2(Sum2 &r, double a, double b) { r.fma2(a, b); }
__device__ __forceinline__ void dot2(Sum2 &r, zd a, zd b) {  // Re(conj(a) b)
    r.fma2(a.x, b.x);
    r.fma2(a.y, b.y);
}
// Over the lanes of a warp, in every lane.
__device__ __forceinline__ Sum2 warp_sum2(Sum2 r) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        r.add(__shfl_xor_sync(0xffffffffu, r.s, o), __shfl_xor_sync(0xffffffffu, r.c, o));
    return r;
}
__host__ __device__ constexpr size_t align16(size_t b) { return (b + 15) / 16 * 16; }

// Shared memory, in this order; the resident columns and entries come last.
template <class C>
struct Layout {
    size_t x, y, v, z, comb, a, ad, tot, sp, ta, tb, red, col, start, count, wide, end;
    __host__ __device__ Layout(int chunk, int kmax) {
        size_t o = 0;
        auto take = [&](size_t bytes) {
            const size_t at = o;
            o += align16(bytes);
            return at;
        };
        x = take(sizeof(C) * chunk);
        y = take(sizeof(C) * chunk);
        v = take(sizeof(C) * chunk);
        z = take(sizeof(C) * chunk);
        comb = take(sizeof(C) * 2 * kThreads);
        a = take(sizeof(C) * (kmax + 1));
        ad = take(sizeof(C) * 2 * (kmax + 1));
        tot = take(sizeof(double) * step_doubles<C>(kmax));
        sp = take(sizeof(double) * step_doubles<C>(kmax));
        ta = take(sizeof(double) * (kmax + 1));
        tb = take(sizeof(double) * (kmax + 1));
        red = take(sizeof(double) * kThreads);
        col = take(sizeof(C *) * (kmax + 1));
        start = take(sizeof(int) * chunk);
        count = take(sizeof(int) * chunk);
        wide = take(sizeof(unsigned short) * chunk);
        end = o;
    }
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The double at p (this block's shared memory) in block `rank` of the cluster.
__device__ __forceinline__ double peer_double(const double *p, unsigned rank) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    unsigned ra;
    double v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(ra) : "memory");
    return v;
}

// Barrier over the grid (all blocks resident: a cooperative launch), after
// the caller's cluster met: one block of a cluster arrives for all, every
// block waits, for at most `polls` looks.  *gave_up is set when that ran out;
// the block goes on without waiting then (its results are not used) and keeps
// meeting its cluster.  It no longer waits for the cluster's first block to
// have read its sums, so it must neither write them again nor end before that.
__device__ __forceinline__ void grid_meet(unsigned *counter, unsigned target, bool arrive, long polls, int *gave_up) {
    __syncthreads();
    if (threadIdx.x == 0) {
        if (arrive) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
        long i = *gave_up ? polls : 0;
        unsigned seen;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
        } while (seen < target && ++i < polls);
        if (seen < target) *gave_up = 1;
    }
    __syncthreads();
}

// Sums of N values (a power of two) over the lanes of a warp, halving the
// values with the lanes: N - 1 + 5 - log2 N shuffles.  The total of value i
// ends in v[0] of the lanes whose upper log2 N bits spell i.
template <int N>
__device__ __forceinline__ void warp_sums(double (&v)[N], int lane) {
    int o = 16;
#pragma unroll
    for (int n = N / 2; n > 0; n /= 2, o /= 2) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const double send = up ? v[i] : v[i + n], mine = up ? v[i + n] : v[i];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    for (; o > 0; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}

template <class C>
__global__ void __launch_bounds__(kThreads, 1) k_coop(const CoopArgs<C> A) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int cw = cwidth<C>();
    const Layout<C> L(A.chunk, A.kmax);
    C *const sx = reinterpret_cast<C *>(smem + L.x), *const sy = reinterpret_cast<C *>(smem + L.y);
    C *const sv = reinterpret_cast<C *>(smem + L.v), *const sz = reinterpret_cast<C *>(smem + L.z);
    C *const comb = reinterpret_cast<C *>(smem + L.comb);
    C *const sa = reinterpret_cast<C *>(smem + L.a);
    C *const ad = reinterpret_cast<C *>(smem + L.ad);  // h and the pass's other coefficient, per column
    double *const tot = reinterpret_cast<double *>(smem + L.tot), *const sp = reinterpret_cast<double *>(smem + L.sp);
    double *const ta = reinterpret_cast<double *>(smem + L.ta), *const tb = reinterpret_cast<double *>(smem + L.tb);
    double *const red = reinterpret_cast<double *>(smem + L.red);
    C **const scol = reinterpret_cast<C **>(smem + L.col);  // the column table, columns 0 .. kmax
    int *const est = reinterpret_cast<int *>(smem + L.start), *const ecn = reinterpret_cast<int *>(smem + L.count);
    unsigned short *const wide = reinterpret_cast<unsigned short *>(smem + L.wide);  // the block's long rows
    C *const vres = reinterpret_cast<C *>(smem + L.end);  // column c, row i at c * chunk + i
    C *const eva = vres + (size_t)A.nres * A.chunk;
    int *const eci = reinterpret_cast<int *>(eva + A.ecap);
    __shared__ int gave_up;
    __shared__ int nwide;
    __shared__ double dd[6];    // |z|^2, Re p_k, g_k in two doubles each
    __shared__ __align__(16) double next[4];  // 1 / beta, beta^2, h_{k-1}
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int W = kThreads / 32;
    constexpr int kProductThreads = kThreads - 64;
    const int bid = blockIdx.x, chunk = A.chunk, nres = A.nres;
    const unsigned cs = cluster_size(), crank = cluster_rank();
    const int NCl = gridDim.x / cs, cid = bid / cs;  // clusters
    const long r0 = (long)bid * chunk;
    const int rows = (int)max(0L, min((long)chunk, A.n_pad - r0));

    // ---- the block's state for the run -----------------------------------
    if (tid == 0) gave_up = 0;
    for (int i = tid; i < A.j0; i += kThreads) {
        ta[i] = A.ta[i];
        tb[i] = A.tb[i];
    }
    for (int i = tid; i <= A.kmax; i += kThreads) scol[i] = A.cols[i];
    const int estride = A.sell ? 32 : 1;
    const long rfirst = min(r0, (long)A.nrow);
    const long long ebase = A.sell ? A.ptr[(rfirst + 31) / 32] : A.ptr[rfirst];
    const long rend = min(r0 + rows, (long)A.nrow);
    const long long elast = rend > r0 ? (A.sell ? A.ptr[(rend + 31) / 32] : A.ptr[rend]) : ebase;
    const int nent = (int)(elast - ebase);
    const bool cached = nent <= A.ecap;
    if (tid == 0) nwide = 0;
    __syncthreads();
    for (int i = tid; i < rows; i += kThreads) {
        const long row = r0 + i;
        int st = 0, cn = 0;
        if (row < A.nrow) {
            if (A.sell) {
                const long long b = A.ptr[row / 32];
                st = (int)(b - ebase) + (int)(row & 31);
                cn = (int)((A.ptr[row / 32 + 1] - b) >> 5);
            } else {
                st = (int)(A.ptr[row] - ebase);
                cn = (int)(A.ptr[row + 1] - A.ptr[row]);
            }
        }
        est[i] = st;
        ecn[i] = cn;
        if (cn > A.wide) wide[atomicAdd(&nwide, 1)] = (unsigned short)i;
        sv[i] = ldcg(A.cols[A.j0] + row);
        sx[i] = sv[i];
    }
    if (cached) {
        for (int e = tid; e < nent; e += kThreads) {
            eva[e] = A.va[ebase + e];
            eci[e] = A.ci[ebase + e];
        }
    }
    // Four columns at a time, to have their loads in flight together.
    for (int c = 0; c < min(nres, A.j0 + 1); c += 4) {
        const int cn = min(4, min(nres, A.j0 + 1) - c);
        const C *src[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) src[u] = A.cols[c + min(u, cn - 1)] + r0;
        for (int i = tid; i < rows; i += kThreads) {
            C t[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) t[u] = ldcg(src[u] + i);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (u < cn) vres[(size_t)(c + u) * chunk + i] = t[u];
        }
    }
    // In the pass column slices.
    const int slices = max(1, kThreads / chunk);
    const int sl = slices > 1 ? tid / chunk : 0;
    __syncthreads();

    const int nw = nwide;
    double sigma = ta[A.j0 - 1], delta = 0.0;
    unsigned meets = 0;
    // Adds the clusters' partial sums of the step that made column k (into
    // tot), forms delta and the new sigma.
    auto close_step = [&](int s) {
        const int k = A.j0 + s - 1, D = step_doubles<C>(k);
        const double *const part = A.part + (size_t)(s & 1) * NCl * step_doubles<C>(A.kmax);
        const int dp = (D + 31) / 32 * 32;
        const int ng = max(1, (kThreads - 96) / dp);  // groups of clusters summed side by side
        if (warp < W - 3) {
            constexpr int U = 10;
            for (int d0 = 0; d0 < D; d0 += kThreads - 96) {
                const int d = d0 + (ng > 1 ? tid % dp : tid), gi = ng > 1 ? tid / dp : 0;
                double sum = 0.0;
                if (d < D && gi < ng) {
                    for (int b0 = gi; b0 < NCl; b0 += U * ng) {
                        double t[U];
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            t[u] = b0 + u * ng < NCl ? __ldcg(part + (size_t)(b0 + u * ng) * D + d) : 0.0;
#pragma unroll
                        for (int u = 0; u < U; ++u) sum += t[u];
                    }
                    if (ng == 1) tot[d] = sum;
                    else red[tid] = sum;
                }
            }
        } else {
            // The sums in two doubles: one warp each.
            const int w = warp - (W - 3);
            Sum2 r;
            for (int b = lane; b < NCl; b += 32) {
                const double *p = part + (size_t)b * D + (D - 6) + 2 * w;
                r.add(__ldcg(p), __ldcg(p + 1));
            }
            r = warp_sum2(r);
            if (lane == 0) {
                dd[2 * w] = r.s;
                dd[2 * w + 1] = r.c;
            }
        }
        __syncthreads();
        if (ng > 1) {
            if (tid < D) {
                double v = red[tid];
                for (int q = 1; q < ng; ++q) v += red[q * dp + tid];
                tot[tid] = v;
            }
            __syncthreads();
        }
        // p / g with g = |q_k|^2, which is 1 to rounding (checked below):
        // 1 / g = 2 - g to the square of that.
        const double g = dd[4] + dd[5];
        delta = (dd[2] + dd[3]) * (2.0 - g);
        sigma += delta;
    };
    // |x|^2 = |z|^2 - 2 delta Re p_k + delta^2 g_k.
    auto norm_x = [&]() {
        Sum2 x;
        x.add(dd[0], dd[1]);
        x.fma2(-2.0 * delta, dd[2]);
        x.c = fma(-2.0 * delta, dd[3], x.c);
        const double d2 = delta * delta, d2e = fma(delta, delta, -d2);
        x.fma2(d2, dd[4]);
        x.c = fma(d2, dd[5], fma(d2e, dd[4], x.c));
        return x.s + x.c;
    };
    // By one warp: h = p - delta g (k values, into sa), returning the
    // arrowhead row of T h.
    auto take_h = [&](int k) {
        const C *const pg = reinterpret_cast<const C *>(tot);  // p, g of column c at 2 c, 2 c + 1
        C arrow = czero(C());
        for (int c = lane; c < k; c += 32) {
            const C h = pg[2 * c] - delta * pg[2 * c + 1];
            sa[c] = h;
            if (c < A.kept) arrow = arrow + tb[c] * h;
        }
        if (A.kept > 0) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) arrow = arrow + shfl_x(arrow, o);
        }
        __syncwarp();
        return arrow;
    };
    // By another: the scalars of step s, logged by the first block; beta^2
    // and 1 / beta for the pass.
    auto take_scalars = [&](int s, int k) {
        const C *const pg = reinterpret_cast<const C *>(tot);
        double h2 = 0.0;
        for (int c = lane; c < k; c += 32) h2 += abs2(pg[2 * c] - delta * pg[2 * c + 1]);
        const double x2 = norm_x();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) h2 += __shfl_xor_sync(0xffffffffu, h2, o);
        const double nb2 = x2 - h2;
        if (lane == 0) {
            next[0] = rsqrt(nb2);
            next[1] = nb2;
            if (bid == 0) {
                double *lg = A.log + 4 * s;
                const bool fine = delta * delta <= 256.0 * x2 && fabs(dd[4] - 1.0) < 1e-8;
                lg[0] = sigma;
                lg[1] = fine ? x2 : nan("");
                lg[2] = h2;
                lg[3] = nb2;  // |r|^2 after the pass
            }
        }
    };
    double ib = 1.0, b2 = 0.0;
    for (int s = 1; s <= A.S; ++s) {
        const int k = A.j0 + s - 1;  // this step finishes column k and projects the next
        if (s > 1) close_step(s - 1);
        if (warp < W - 2) {
            // ---- y = A x on the block's rows; x = z - delta q_{k-1} ------------
            // (the first product is of column j0 itself: delta is zero)
            const C *const gz = s > 1 ? A.z[(s - 1) & 1] : scol[A.j0];
            const C *const gv = scol[k - (s > 1 ? 1 : 0)];
            const double dl = delta;
            const C *va = cached ? eva : A.va + ebase;
            const int *ci = cached ? eci : A.ci + ebase;
            // 2^A.lanes lanes per row; then the long rows, a warp each.
            for (int turn = 0; turn < (nw > 0 ? 2 : 1); ++turn) {
                const int lg = turn ? 5 : A.lanes, lanes = 1 << lg, items = turn ? nw : rows, sub = tid & (lanes - 1);
                for (int i0 = 0; i0 < items; i0 += kProductThreads >> lg) {
                    const int e = i0 + (tid >> lg), i = e < items ? (turn ? wide[e] : e) : 0;
                    const int st = est[i], cn = ecn[i];
                    const bool on = e < items && (turn || cn <= A.wide);
                    C acc = czero(C());
                    if (on) {
                        constexpr int U = 8 / cw;
                        for (int t0 = sub; t0 < cn; t0 += U * lanes) {
                            C xz[U], xv[U];
#pragma unroll
                            for (int u = 0; u < U; ++u) {
                                if (t0 + u * lanes < cn) {
                                    const int col = ci[st + (t0 + u * lanes) * estride];
                                    xz[u] = ldcg(gz + col);
                                    xv[u] = ldcg(gv + col);
                                }
                            }
#pragma unroll
                            for (int u = 0; u < U; ++u)
                                if (t0 + u * lanes < cn)
                                    acc = acc + mulx(va[st + (t0 + u * lanes) * estride], xz[u] - dl * xv[u]);
                        }
                    }
                    for (int o = lanes / 2; o > 0; o >>= 1) acc = acc + shfl_x(acc, o);
                    if (sub == 0 && on) {
                        sy[i] = acc;
                        if (s > 1) sx[i] = sz[i] - dl * sv[i];
                    }
                }
            }
        } else if (s == 1) {
            // A finished vector: only the recurrence (the arrowhead row of a
            // restart, or the column before).
            if (warp == W - 1) {
                for (int i = lane; i < k; i += 32) {
                    ad[2 * i] = czero(C());
                    ad[2 * i + 1] = as_c(A.kept == A.j0 || i == k - 1 ? tb[i] : 0.0, C());
                }
                if (lane == 0) {
                    next[0] = 1.0;
                    next[1] = 0.0;
                    *reinterpret_cast<C *>(next + 2) = czero(C());
                }
            }
        } else if (warp == W - 2) {
            take_scalars(s - 1, k);
        } else {
            // ---- the pass's coefficients: h, and T h - (sigma + h_{k-1}) h ---------
            // (beta^2 of the recurrence is added in the pass)
            const C arrow = take_h(k);
            const C hl = sa[k - 1];
            if (lane == 0) {
                ta[k - 1] = sigma;
                if (s > 2) tb[k - 2] = sqrt(b2);  // the beta before this step's
                *reinterpret_cast<C *>(next + 2) = hl;
            }
            __syncwarp();
            const C shift = as_c(sigma, C()) + hl;
            for (int i = lane; i < k; i += 32) {
                C c = ta[i] * sa[i];
                if (i < A.kept) {
                    c = c + tb[i] * sa[A.kept];
                } else {
                    if (i > A.kept)
                        c = c + tb[i - 1] * sa[i - 1];
                    else
                        c = c + arrow;
                    if (i + 1 < k) c = c + tb[i] * sa[i + 1];
                }
                ad[2 * i] = sa[i];
                ad[2 * i + 1] = c - mulx(shift, sa[i]);
            }
        }
        __syncthreads();
        ib = next[0];
        b2 = next[1];
        // ---- q_k and z on the block's rows ---------------------------------------
        const C shift = as_c(sigma, C()) + *reinterpret_cast<const C *>(next + 2);
        C *const zout = A.z[s & 1];
        C *const vk = scol[k];
        for (int i0 = 0; i0 < rows; i0 += kThreads) {
            const int i = slices > 1 ? tid - sl * chunk : i0 + tid;
            const bool on = sl < slices && i < rows;
            C u = czero(C()), w = czero(C()), u1 = czero(C()), w1 = czero(C());
            if (on) {
                // Two sums of each kind, for shorter chains.
                int c = sl;
                const int kr = min(k, nres);
#pragma unroll 4
                for (; c + slices < kr; c += 2 * slices) {
                    const C e = vres[(size_t)c * chunk + i], f = vres[(size_t)(c + slices) * chunk + i];
                    fma_c(u, e, ad[2 * c]);
                    fma_c(w, e, ad[2 * c + 1]);
                    fma_c(u1, f, ad[2 * (c + slices)]);
                    fma_c(w1, f, ad[2 * (c + slices) + 1]);
                }
                if (c < kr) {
                    const C e = vres[(size_t)c * chunk + i];
                    fma_c(u, e, ad[2 * c]);
                    fma_c(w, e, ad[2 * c + 1]);
                    c += slices;
                }
#pragma unroll 8
                for (; c < k; c += slices) {
                    const C e = scol[c][r0 + i];
                    fma_c(u, e, ad[2 * c]);
                    fma_c(w, e, ad[2 * c + 1]);
                }
                u = u + u1;
                w = w + w1;
            }
            if (slices > 1) {
                comb[2 * tid] = u;
                comb[2 * tid + 1] = w;
                __syncthreads();
                if (on && sl == 0) {
                    for (int q = 1; q < slices; ++q) {
                        u = u + comb[2 * (tid + q * chunk)];
                        w = w + comb[2 * (tid + q * chunk) + 1];
                    }
                }
            }
            if (on && sl == 0) {
                const C x = sx[i];
                const C q = ib * (x - u);
                const C z = ib * ((sy[i] - mulx(shift, x)) - (w + b2 * sv[i]));  // sv: q_{k-1} still
                sv[i] = q;
                sz[i] = z;
                if (s > 1) {
                    vk[r0 + i] = q;
                    if (k < nres) vres[(size_t)k * chunk + i] = q;
                }
                zout[r0 + i] = z;
            }
            if (slices > 1) break;  // one round covers the chunk
        }
        __syncthreads();
        // ---- partial p, g of every column (most warps); |z|^2, Re p_k, g_k ------
        // (not over sums that the cluster's first block may still be reading)
        const int D = step_doubles<C>(k);
        if (gave_up) {
        } else if (warp < W - 3) {
            constexpr int NCW = 4 / cw;         // columns per warp and round
            constexpr int NV = 2 * cw * NCW;
            for (int c0 = warp * NCW; c0 <= k; c0 += (W - 3) * NCW) {
                const C *v[NCW];
                C p[NCW], g[NCW];
#pragma unroll
                for (int u = 0; u < NCW; ++u) {
                    const int c = c0 + u;
                    v[u] = c < k ? (c < nres ? vres + (size_t)c * chunk : scol[c] + r0) : sv;
                    p[u] = g[u] = czero(C());
                }
#pragma unroll 2
                for (int i = lane; i < rows; i += 32) {
                    const C zi = sz[i], qi = sv[i];
                    C e[NCW];
#pragma unroll
                    for (int u = 0; u < NCW; ++u) e[u] = v[u][i];
#pragma unroll
                    for (int u = 0; u < NCW; ++u) {
                        fma_conj(p[u], e[u], zi);
                        fma_conj(g[u], e[u], qi);
                    }
                }
                double val[NV];  // in the order of the partial sums
#pragma unroll
                for (int u = 0; u < NCW; ++u) {
                    const double *ps = reinterpret_cast<const double *>(&p[u]);
                    const double *gs = reinterpret_cast<const double *>(&g[u]);
#pragma unroll
                    for (int q = 0; q < cw; ++q) {
                        val[2 * cw * u + q] = ps[q];
                        val[2 * cw * u + cw + q] = gs[q];
                    }
                }
                warp_sums<NV>(val, lane);
                constexpr int kLanes = 32 / NV;  // lanes that hold the same total
                const int idx = lane / kLanes, d = 2 * cw * c0 + idx;
                if (lane % kLanes == 0 && d < 2 * cw * (k + 1)) sp[d] = val[0];
            }
        } else {
            const int w = warp - (W - 3);
            const C *const l = w == 0 ? sz : sv, *const r = w == 2 ? sv : sz;
            Sum2 t;
            for (int i = lane; i < rows; i += 32) dot2(t, l[i], r[i]);
            t = warp_sum2(t);
            if (lane == 0) {
                sp[D - 6 + 2 * w] = t.s;
                sp[D - 5 + 2 * w] = t.c;
            }
        }
        // ---- the cluster's sums, by its first block --------------------------------
        cluster_meet();
        if (crank == 0) {
            double *const po = A.part + (size_t)(s & 1) * NCl * step_doubles<C>(A.kmax) + (size_t)cid * D;
            // (clusters have at most 8 blocks; the loads before the sums)
            for (int d = tid; d < D - 6; d += kThreads) {
                double t[8];
#pragma unroll
                for (unsigned q = 0; q < 8; ++q) t[q] = q < cs ? peer_double(sp + d, q) : 0.0;
#pragma unroll
                for (unsigned q = 1; q < 8; ++q) t[0] += t[q];
                po[d] = t[0];
            }
            if (tid >= kThreads - 3) {
                const int d = D - 6 + 2 * (tid - (kThreads - 3));
                double v[8], e[8];
#pragma unroll
                for (unsigned q = 0; q < 8; ++q) {
                    v[q] = q < cs ? peer_double(sp + d, q) : 0.0;
                    e[q] = q < cs ? peer_double(sp + d + 1, q) : 0.0;
                }
                Sum2 t;
#pragma unroll
                for (unsigned q = 0; q < 8; ++q) t.add(v[q], e[q]);
                po[d] = t.s;
                po[d + 1] = t.c;
            }
        }
        grid_meet(A.sync, ++meets * (unsigned)NCl, crank == 0, A.polls, &gave_up);
    }
    // ---- the last vector ------------------------------------------------------
    {
        const int k = A.j0 + A.S - 1;
        close_step(A.S);
        if (warp == W - 1) take_h(k + 1);
        if (warp == W - 2) take_scalars(A.S, k + 1);
        __syncthreads();
        const double sc = next[0];
        C *const out = scol[k + 1];
        for (int i = tid; i < rows; i += kThreads) {
            C u = czero(C());
            int c = 0;
#pragma unroll 8
            for (; c < min(k, nres); ++c) fma_c(u, vres[(size_t)c * chunk + i], sa[c]);
#pragma unroll 8
            for (; c < k; ++c) fma_c(u, scol[c][r0 + i], sa[c]);
            fma_c(u, sv[i], sa[k]);
            out[r0 + i] = sc * ((sz[i] - delta * sv[i]) - u);
        }
    }
    if (gave_up && tid == 0) *A.failed = 1.0;  // the host takes no step of the run
    cluster_meet();  // no block ends while its cluster's first may be reading its sums
    // The last block out leaves the counters at zero.
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(A.sync + 1, 1u) == (unsigned)gridDim.x - 1) {
            A.sync[0] = 0;
            A.sync[1] = 0;
        }
    }
}

constexpr size_t kMaxSmem = 220 * 1024;

// How a run over `n_pad` rows and up to `kmax` columns is split.
struct Plan {
    int cluster, chunk, grid, nres, ecap;
    size_t smem;
};

void set_cluster(cudaLaunchAttribute (&attr)[2], int blocks) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
}

// False where the kernel does not apply: operator form, device, sizes.
template <class C>
bool make_plan(const trlx_operator *A, long n_pad, int kmax, size_t part_doubles, Plan *p) {
    if (!A || op_complex(A) != (sizeof(C) == 16) || (op_sell(A) && A->perm)) return false;
    // Per device, set up once: blocks of clusters of 8 and of 4 that are
    // resident together, one per SM (-1: no cooperative launch).  Host threads
    // take turns: none sees a device half set up.
    static std::mutex turn;
    static int blocks_of[64][2] = {};
    int blocks[2];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return false;
    {
        std::lock_guard<std::mutex> hold(turn);
        if (blocks_of[dev][0] == 0) {
            int coop = 0;
            cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
            if (cudaFuncSetAttribute(k_coop<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) !=
                cudaSuccess)
                coop = 0;
            cudaLaunchAttribute attr[2];
            cudaLaunchConfig_t cfg = {};
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = kMaxSmem;
            cfg.attrs = attr;
            cfg.numAttrs = 2;
            for (int i = 0; i < 2; ++i) {
                const int cs = i == 0 ? 8 : 4;
                set_cluster(attr, cs);
                cfg.gridDim = dim3(cs);
                int n = 0;
                if (!coop || cudaOccupancyMaxActiveClusters(&n, k_coop<C>, &cfg) != cudaSuccess) n = 0;
                blocks_of[dev][i] = n > 0 ? n * cs : -1;
            }
            cudaGetLastError();
        }
        blocks[0] = blocks_of[dev][0];
        blocks[1] = blocks_of[dev][1];
    }
    // Clusters of 8 while their blocks keep 256 rows or fewer; of 4, which
    // cover more SMs, for longer vectors.
    int cs = 8, most = blocks[0];
    if (most < 0 || n_pad > 256L * most) {
        cs = 4;
        most = blocks[1];
    }
    if (most < cs) return false;
    const long chunk = ((n_pad + most - 1) / most + 31) / 32 * 32;
    p->cluster = cs;
    p->chunk = (int)chunk;
    p->grid = (int)(((n_pad + chunk - 1) / chunk + cs - 1) / cs * cs);
    const Layout<C> L((int)chunk, kmax);
    if (L.end > kMaxSmem) return false;
    if ((size_t)2 * (p->grid / cs) * step_doubles<C>(kmax) > part_doubles) return false;
    // Entries of a block in shared memory up to a third of what is left
    // (twice the average, for uneven rows), basis columns in the rest.
    const size_t left = kMaxSmem - L.end;
    const size_t per = sizeof(C) + sizeof(int);
    const size_t ecap = std::min<size_t>(left / 3 / per, (size_t)(2 * (A->nnz / p->grid + 1) + 64)) / 4 * 4;
    p->nres = (int)std::min<size_t>((left - ecap * per) / (sizeof(C) * chunk), (size_t)kmax);
    p->ecap = (int)ecap;
    p->smem = L.end + (size_t)p->nres * chunk * sizeof(C) + ecap * per;
    return true;
}

}  // namespace

template <class C>
bool coop_pays(const trlx_operator *A, long n_pad) {
    const long long words = cwidth<C>() * A->nnz;
    return n_pad < kCoopRows && (words <= kCoopWords || words < (op_sell(A) ? 16384ll : 512ll) * A->longest);
}

template <class C>
bool coop_applies(const trlx_operator *A, long n_pad, int kmax, size_t part_doubles) {
    Plan p;
    return make_plan<C>(A, n_pad, kmax, part_doubles, &p);
}

template <class C>
int launch_coop(const trlx_operator *A, C *const *cols, C *z0, C *z1, long n_pad, int j0, int S, int kept,
                const double *ta, const double *tb, double *log, double *failed, double *part, size_t part_doubles,
                unsigned *sync, long polls, cudaStream_t st) {
    Plan p;
    if (S < 1 || j0 < 1 || !make_plan<C>(A, n_pad, j0 + S, part_doubles, &p)) return -1;
    CoopArgs<C> a;
    a.kmax = j0 + S;
    a.nres = p.nres;
    a.ecap = p.ecap;
    a.nrow = A->nrow;
    a.n_pad = n_pad;
    a.chunk = p.chunk;
    // Lanes per row: one while a row's entries are loaded together anyway
    // (neighbouring rows of a lattice then read neighbouring values).
    a.lanes = 0;
    while (a.lanes < 5 && A->nnz > (8ll << a.lanes) * A->nrow) ++a.lanes;
    a.sell = op_sell(A) ? 1 : 0;
    // A row of more than four such loads gets a warp: the other rows, and with
    // them the grid, would wait for it (lattice with one row of 3000 entries,
    // 30000 rows, a call: 49.5 -> 4.8 ms; of 300, 7.6 -> 3.0; discrete kernels
    // 14.3 and 7.3).  Not in SELL form, where 32 neighbouring rows are as long.
    a.wide = a.sell || a.lanes == 5 ? INT_MAX : 32 << a.lanes;
    a.ptr = a.sell ? A->slice_ptr : A->row_ptr;
    a.ci = A->col;
    a.va = static_cast<const C *>(A->val);
    a.cols = cols;
    a.z[0] = z0;
    a.z[1] = z1;
    a.j0 = j0;
    a.S = S;
    a.kept = kept;
    a.ta = ta;
    a.tb = tb;
    a.log = log;
    a.failed = failed;
    a.part = part;
    a.sync = sync;
    a.polls = polls;
    cudaLaunchAttribute attr[2];
    set_cluster(attr, p.cluster);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    if (cudaLaunchKernelEx(&cfg, k_coop<C>, a) == cudaSuccess) return 0;
    cudaGetLastError();
    return -1;
}

template bool coop_pays<double>(const trlx_operator *, long);
template bool coop_pays<zd>(const trlx_operator *, long);
template bool coop_applies<double>(const trlx_operator *, long, int, size_t);
template bool coop_applies<zd>(const trlx_operator *, long, int, size_t);
template int launch_coop<double>(const trlx_operator *, double *const *, double *, double *, long, int, int, int,
                                 const double *, const double *, double *, double *, double *, size_t, unsigned *,
                                 long, cudaStream_t);
template int launch_coop<zd>(const trlx_operator *, zd *const *, zd *, zd *, long, int, int, int, const double *,
                             const double *, double *, double *, double *, size_t, unsigned *, long,
                             cudaStream_t);

}  // namespace trlb
