// Single-sweep Lanczos steps.
//
// A Lanczos step orthogonalises r = A q_{k-1} - alpha q_{k-1} - beta q_{k-2}
// against the basis V (k columns): h = V^H r, r <- r - V h, q_k = r / |r|.
// Done as two kernels, the projection and the update each stream the whole
// basis, and at long vectors that is all a step costs.  The update of one
// step and the projection of the next can share a pass: the operator is
// applied to the vector before its update, y = A r, and corrected afterwards
// with the Lanczos relation A V = V T + beta q_k e_{k-1}^T,
//
//   q_k   = (r - V h) / beta
//   A q_k = (y - V T h) / beta - h_{k-1} q_k
//   r'    = A q_k - alpha q_k - beta q_{k-1}
//
// where beta^2 = |r|^2 - |h|^2 (exact to rounding: the caller accepts a step
// only when |h|^2 < eps |r|^2) and alpha = Re(r^H y) / beta^2 - 2 Re h_{k-1}
// are known before the pass.  Each row needs two sums over the columns (V h
// and V c) before its entries of q_k and r' exist, and then enters the next
// projection h' = [V q_k]^H r'.  One pass reads V, r and y once and writes
// q_k and r'; the corrections are of the size of h, so every quantity is as
// accurate as in the two-kernel step.
//
// Bound by memory; measured against the two kernels and the normalisation
// (one B200): 256^3 FP64, 128 steps, 427 -> 249 ms a call (the sweeps at
// 5.9-6.0 TB/s); 1024^2 complex128, 64.3 -> 38.8 ms; 101^3 FP32, 30.3 -> 17.0
// ms; 2048^2 complex64, 82.4 -> 64.8 ms (12 FP64 FMAs and four conversions per
// 8 bytes: the sweep itself runs at 3.7-3.9 TB/s there).
//
// A sweep takes at most 128 columns: in a larger basis the steps from there on
// read the basis twice (the discrete kernels).
//
// For a 32-bit basis the working vectors stay FP64: q_{k-1} is read from its
// FP64 copy, V T h is formed from the stored columns (h is then of the size
// of the storage rounding, and its error of that size squared).
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "sweep.h"

namespace trlb {

namespace {

constexpr int kWarps = 8, kCols = 16;
constexpr int kNT = kWarps * 32;
static_assert(kWarps * kCols == kSweepCols, "columns of a sweep");
constexpr int kTicketSweep = 4;
constexpr size_t kSmemMax = 221 * 1024;  // dynamic shared memory of a sweep

// A sweep over G groups of at most NC columns.  Shared memory: a ring of
// kStages stages (per warp a tile of NC x 512 bytes, per slice a tile of x
// and y, for 32-bit storage of q_{k-1} too) and one tile of r' per slice.
template <class T, int NC, int G>
struct Shape {
    using C = typename Store<T>::C;
    static constexpr int kSlices = kWarps / G, kRows = 32 * Store<T>::R;
    static constexpr int kVecs = sizeof(T) == sizeof(C) ? 2 : 3;
    static constexpr int kVec = kRows * (int)sizeof(C);  // bytes of one vector's tile
    static constexpr int kSlot = NC * 512;               // bytes of one warp's tile
    static constexpr int kStage = kWarps * kSlot + kSlices * kVecs * kVec;
    // A tile stays in registers between its two phases, except 16 complex64
    // columns per warp, which spill (382 against 347 us at 2^20 rows, 128
    // columns): they are read again, and the partial sums have room of their
    // own.  (Held is better where it fits: complex64, 96 columns, 263 against
    // 295 us; FP32, 2^21 rows, 128 columns, 259 against 295 us.)
    static constexpr bool kHold = !(std::is_same<T, zf>::value && NC == 16);
    static constexpr int kPart = kHold ? 0 : kRows * 2 * (int)sizeof(C);  // bytes per warp
    static constexpr int kTail = kSlices * kVec + kWarps * kPart;
    static constexpr int kFit = (int)((kSmemMax - kTail) / kStage);
    static constexpr int kStages = kFit < 6 ? kFit : 6;
    static_assert(kStages >= 2, "a tile in flight while one is used");
    static constexpr size_t kSmem = (size_t)kStages * kStage + kTail;
};

__device__ __forceinline__ double cmul(double a, double b) { return a * b; }
__device__ __forceinline__ zd cmul(zd a, zd b) { return zd{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__device__ __forceinline__ double shfl_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ zd shfl_xor(zd v, int o) {
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

// The R elements of 16 staged bytes.
__device__ __forceinline__ void unpack(const uint4 &w, double (&o)[2]) {
    o[0] = __hiloint2double((int)w.y, (int)w.x);
    o[1] = __hiloint2double((int)w.w, (int)w.z);
}
__device__ __forceinline__ void unpack(const uint4 &w, double (&o)[4]) {
    o[0] = __uint_as_float(w.x);
    o[1] = __uint_as_float(w.y);
    o[2] = __uint_as_float(w.z);
    o[3] = __uint_as_float(w.w);
}
__device__ __forceinline__ void unpack(const uint4 &w, zd (&o)[1]) {
    o[0] = zd{__hiloint2double((int)w.y, (int)w.x), __hiloint2double((int)w.w, (int)w.z)};
}
__device__ __forceinline__ void unpack(const uint4 &w, zd (&o)[2]) {
    o[0] = zd{__uint_as_float(w.x), __uint_as_float(w.y)};
    o[1] = zd{__uint_as_float(w.z), __uint_as_float(w.w)};
}

// The columns are cut into G groups (G the smallest power of two with
// 16 G >= k) of NC - 2 to NC columns; the 8 / G warps of a group take
// alternate row tiles (slices) of 32 R rows, so every warp streams at every
// basis size.  Each lane copies its own 16 bytes of each of its warp's
// columns into a ring by cp.async (all stages but the one in use in flight,
// 128 KB per SM or more; one block per SM) and holds the tile in registers
// through the two phases of a tile:
//   1. partial sums of V h and V c over the warp's columns, left in the
//      ring slot just read; the G warps of the slice meet; up to four lanes
//      per row add the G partials and form q_k and r' (x, y loaded one tile
//      ahead);
//   2. the warps meet again and add conj(V) r' to their column sums.
// Eight warps of 16 columns rather than 16 of 8: half the partial sums and
// barrier traffic per tile, and registers for the coefficients of real types.
template <class T, int NC, int G>
__global__ void __launch_bounds__(kNT, 1) k_sweep(const SweepArgs<T> A, long chunk, typename Store<T>::C *part,
                                                  double *part_r2, unsigned *ticket) {
    using S = Store<T>;
    using C = typename S::C;
    using Sh = Shape<T, NC, G>;
    constexpr int R = S::R, NS = Sh::kStages, wpg = Sh::kSlices;
    constexpr bool kWide = sizeof(T) == sizeof(C);
    constexpr bool kHold = Sh::kHold;
    constexpr bool kCoefRegs = std::is_same<T, double>::value;  // FP64 leaves registers for them
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ C coef[G * NC][2];  // of column q of group g at g * NC + q
    __shared__ C red_c[kWarps][NC];
    __shared__ C red_s[32];
    __shared__ double red_d[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k = A.k;
    // Group g has k / G columns, one more for g < k % G: NC - 2 to NC (a
    // single group of fewer repeats its last column with zero coefficients).
    const int few = k / G, more = k - few * G;
    const int grp = warp / wpg, slice = warp - grp * wpg;
    auto first_col = [&](int gg) { return gg * few + min(gg, more); };
    const int cb = first_col(grp), cn = few + (grp < more ? 1 : 0);
    const bool on1 = cn >= NC - 1 || G == 1, on0 = cn >= NC || G == 1;  // the last two columns
    auto on = [&](int q) { return q < NC - 2 || (q == NC - 2 ? on1 : on0); };
    const long row0 = (long)blockIdx.x * chunk, row1 = min(A.n_pad, row0 + chunk);
    const int tiles = row1 > row0 ? (int)((row1 - row0) / Sh::kRows) : 0;
    const int nit = tiles > slice ? (tiles - slice + wpg - 1) / wpg : 0;
    // The slice's tiles, upwards for even k and downwards for odd: what L2
    // (126 MB) still holds of the last sweep's rows is read first.  1024^2
    // complex128, 64 MB to 2 GB a sweep: 45.8 -> 41.7 ms a call; 101^3 FP32:
    // 19.1 -> 18.0 ms; 64^3 FP64: 13.7 -> 13.5 ms.
    constexpr int kStep = wpg * Sh::kRows;
    const bool down = (k & 1) != 0;
    const int step = down ? -kStep : kStep;  // rows from tile to tile
    const long tile0 = row0 + (long)slice * Sh::kRows + (down ? (long)max(nit - 1, 0) * kStep : 0L);
    // This lane's next copies: `from` plus each column's offset in the pool,
    // in 16-byte units (one multiply-add per copy, one register per column).
    const char *const pool = reinterpret_cast<const char *>(A.pool);
    const char *from = pool + (size_t)(tile0 + lane * R) * sizeof(T);
    unsigned off[NC];
#pragma unroll
    for (int q = 0; q < NC; ++q)
        off[q] = (unsigned)((reinterpret_cast<const char *>(A.cols[min(cb + q, k - 1)]) - pool) >> 4);
    // The slice's vector tiles, 512 bytes per warp and copy.
    constexpr int kVecCopies = Sh::kVecs * Sh::kVec / 512, kPerVec = Sh::kVec / 512;
    long vrow = tile0;
    int issued = 0;
    unsigned ifill = 0, iuse = 0;  // byte offsets of the stages to fill and to use
    auto next_stage = [](unsigned o) { return o == (unsigned)((NS - 1) * Sh::kStage) ? 0u : o + Sh::kStage; };
    auto fill_cols = [&]() {
        if (issued < nit) {
            unsigned char *d = smem + ifill + warp * Sh::kSlot + lane * 16;
#pragma unroll
            for (int q = 0; q < NC; ++q)
                if (on(q)) cp_async16(d + q * 512, from + (size_t)off[q] * 16);
            from += (long)step * (int)sizeof(T);
        }
    };
    auto fill_vecs = [&]() {
        if (issued < nit) {
            unsigned char *dv = smem + ifill + kWarps * Sh::kSlot + slice * Sh::kVecs * Sh::kVec + lane * 16;
#pragma unroll
            for (int j = 0; j < kVecCopies; ++j) {
                if (j % G == grp) {
                    const C *src = j / kPerVec == 0 ? A.x : (j / kPerVec == 1 ? A.y : A.xp);
                    cp_async16(dv + j * 512,
                               reinterpret_cast<const char *>(src + vrow) + (j % kPerVec) * 512 + lane * 16);
                }
            }
            vrow += step;
        }
    };
    auto filled = [&]() {
        ++issued;
        ifill = next_stage(ifill);
    };
    auto issue = [&]() {
        fill_cols();
        fill_vecs();
        cp_async_commit();
        filled();
    };
    // The kernel may start before the operator's (launch_sweep): the basis is
    // older than that one, the vectors and the scalars are read after it.
#pragma unroll
    for (int t = 0; t < NS - 1; ++t) {
        fill_cols();
        filled();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    issued = 0;
    ifill = 0;
#pragma unroll
    for (int t = 0; t < NS - 1; ++t) {
        fill_vecs();
        cp_async_commit();
        filled();
    }
    const double ib = A.sc[0], b2 = A.sc[1], rbeta = kWide ? 0.0 : A.sc[2];
    const C hl = A.a[k - 1];
    const double alpha = *A.dot / b2 - 2.0 * real_part(hl);
    const C g = as_c(alpha, C()) + hl;
    for (int e = tid; e < G * NC; e += kNT) {
        const int gg = e / NC, q = e - gg * NC, c = first_col(gg) + q;
        const bool in = q < few + (gg < more ? 1 : 0);
        const C ac = in ? A.a[c] : czero(C());
        coef[e][0] = ac;
        coef[e][1] = in ? A.c[c] - cmul(g, ac) : czero(C());
    }
    T *const vk = A.cols[k];
    // Rows of a tile for the middle part: with G >= R, tpr lanes of a warp
    // per row (32 / tpr rows per warp); else R / G rows per lane.
    constexpr int tpr = G >= 4 * R ? 4 : (G >= 2 * R ? 2 : 1);
    constexpr int rpt = G >= R ? 1 : R / G;
    constexpr int rpw = 32 / tpr;
    const int sub = lane / rpw;
    const int row_l = G >= R ? grp * rpw + (lane - sub * rpw) : grp * 32 + lane;
    const bool owner = row_l < Sh::kRows;
    C *const rbuf = reinterpret_cast<C *>(smem + (size_t)NS * Sh::kStage + slice * Sh::kVec);
    unsigned char *const parts = smem + (size_t)NS * Sh::kStage + wpg * Sh::kVec;
    auto meet = [&]() {
        if (G == 1)
            __syncwarp();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slice), "n"(G * 32) : "memory");
    };
    C acc[NC], qacc = czero(C());
    double r2acc = 0.0;
#pragma unroll
    for (int q = 0; q < NC; ++q) acc[q] = czero(C());
    __syncthreads();
    const C(*const cf)[2] = coef + grp * NC;
    C cr[kCoefRegs ? NC : 1][2];
    if constexpr (kCoefRegs) {
#pragma unroll
        for (int q = 0; q < NC; ++q) {
            cr[q][0] = cf[q][0];
            cr[q][1] = cf[q][1];
        }
    }
    long row = tile0 + row_l;  // this lane's row of the current tile
    for (int t = 0; t < nit; ++t, row += step) {
        issue();  // into the stage whose partials were read at t - 1
        cp_async_wait<NS - 1>();
        unsigned char *const slot = smem + iuse + warp * Sh::kSlot;
        auto tile16 = [&](int q) {
            return on(q) ? *reinterpret_cast<const uint4 *>(slot + q * 512 + lane * 16) : make_uint4(0u, 0u, 0u, 0u);
        };
        uint4 v[kHold ? NC : 1];
        C u[R], w[R];
#pragma unroll
        for (int q = 0; q < R; ++q) u[q] = w[q] = czero(C());
        if constexpr (kHold) {
#pragma unroll
            for (int q = 0; q < NC; ++q) v[q] = tile16(q);
        }
#pragma unroll
        for (int q = 0; q < NC; ++q) {
            const C ca = kCoefRegs ? cr[kCoefRegs ? q : 0][0] : cf[q][0];
            const C cc = kCoefRegs ? cr[kCoefRegs ? q : 0][1] : cf[q][1];
            C e[R];
            unpack(kHold ? v[kHold ? q : 0] : tile16(q), e);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                fma_c(u[i], e[i], ca);
                fma_c(w[i], e[i], cc);
            }
        }
        if (kHold) __syncwarp();  // every lane has read its part of the slot
        {
            C *o = reinterpret_cast<C *>(kHold ? slot : parts + warp * Sh::kPart) + lane * R * 2;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                o[2 * i] = u[i];
                o[2 * i + 1] = w[i];
            }
        }
        meet();
        if (owner) {
            constexpr int kWarpPart = kHold ? Sh::kSlot : Sh::kPart;
            const unsigned char *const sl0 = (kHold ? smem + iuse : parts) + slice * kWarpPart;
            const C *const xs =
                reinterpret_cast<const C *>(smem + iuse + kWarps * Sh::kSlot + slice * Sh::kVecs * Sh::kVec);
#pragma unroll
            for (int i = 0; i < rpt; ++i) {
                const int rl = row_l + i * 32 * G;
                C us = czero(C()), ws = czero(C());
#pragma unroll
                for (int j = 0; j < (G + tpr - 1) / tpr; ++j) {
                    const C *o =
                        reinterpret_cast<const C *>(sl0 + (size_t)((sub + j * tpr) * wpg) * kWarpPart) + rl * 2;
                    us = us + o[0];
                    ws = ws + o[1];
                }
                if (tpr >= 2) {
                    us = us + shfl_xor(us, 16);
                    ws = ws + shfl_xor(ws, 16);
                }
                if (tpr == 4) {
                    us = us + shfl_xor(us, 8);
                    ws = ws + shfl_xor(ws, 8);
                }
                const C xv = xs[rl];
                C q = ib * (xv - us);
                C rn = ib * ((xs[Sh::kRows + rl] - cmul(g, xv)) - ws);
                if (!kWide) rn = rn - rbeta * xs[2 * Sh::kRows + rl];
                if (sub == 0) {
                    const long rg = row + i * 32 * G;
                    rbuf[rl] = rn;
                    if (!A.first) {
                        A.x[rg] = q;
                        if (!kWide) vk[rg] = S::from_c(q);
                    }
                    A.y[rg] = rn;
                    if (!kWide) q = S::to_c(S::from_c(q));
                    fma_conj(qacc, q, rn);
                    r2acc += abs2(rn);
                }
            }
        }
        iuse = next_stage(iuse);
        meet();
        C rv[R];
#pragma unroll
        for (int i = 0; i < R; ++i) rv[i] = rbuf[lane * R + i];
#pragma unroll
        for (int q = 0; q < NC; ++q) {
            C e[R];
            unpack(kHold ? v[kHold ? q : 0] : tile16(q), e);
#pragma unroll
            for (int i = 0; i < R; ++i) fma_conj(acc[q], e[i], rv[i]);
        }
    }
    cp_async_wait<0>();
    // Block partials: each column over its group's warps, then q_k^H r' and
    // |r'|^2; the last block forms the totals and the next sweep's inputs.
    const int m = k + 1;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[q] = acc[q] + shfl_down(acc[q], o);
        if (lane == 0) red_c[warp][q] = acc[q];
    }
    __syncthreads();
    if (tid < G * NC) {
        const int gg = tid / NC, q = tid - gg * NC, c = first_col(gg) + q;
        if (q < few + (gg < more ? 1 : 0)) {
            C s = czero(C());
            for (int sl = 0; sl < wpg; ++sl) s = s + red_c[gg * wpg + sl][q];
            part[(long)blockIdx.x * m + c] = s;
        }
    }
    const C qs = block_sum(qacc, red_s);
    const double rs = block_sum(r2acc, red_d);
    if (tid == 0) {
        part[(long)blockIdx.x * m + k] = qs;
        part_r2[blockIdx.x] = rs;
    }
    if (!last_block_arrived(ticket)) return;
    // Totals, T h and the scalars, one column per thread (k + 1 <= 129 of
    // them).  A thread's loads are all in flight at once; with eight at a
    // time, and one thread alone for |h|^2 and for the coupled row, every
    // sweep took 7 to 30 us longer (FP64, 2^21 rows, 4 and 128 columns: 35.8
    // and 437.8 -> 28.1 and 410.0 us; 64^3 FP64 13.5 -> 12.2 ms a call).
    const int per = kNT / m, col = tid % m, part_of = tid / m;
    // Row tid of T: diagonal, coupling to the next and to the last column
    // (the new entries are stored below).
    const double bprev = sqrt(b2);
    auto tb = [&](int i) { return i == k - 1 && !A.first ? bprev : A.tb[i]; };
    const double ti = tid < k ? A.ta[tid] : alpha, bi = tid < k ? tb(tid) : 0.0;
    const double bl = tid >= 1 && tid <= k ? tb(tid - 1) : 0.0;
    C sum = czero(C());
    if (part_of < per) {
        constexpr int U = 32;
        for (int b0 = part_of; b0 < (int)gridDim.x; b0 += U * per) {
            C v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int b = b0 + u * per;
                v[u] = b < (int)gridDim.x ? ldcg(part + (long)b * m + col) : czero(C());
            }
#pragma unroll
            for (int o = U / 2; o > 0; o >>= 1)
#pragma unroll
                for (int u = 0; u < o; ++u) v[u] = v[u] + v[u + o];
            sum = sum + v[0];
        }
    }
    C *const tot = reinterpret_cast<C *>(smem), *const hs = tot + kNT;
    tot[tid] = sum;
    __syncthreads();
    C hi = czero(C());
    if (tid < m) {
        for (int q = 0; q < per; ++q) hi = hi + tot[q * m + tid];
        A.a[tid] = hi;
        hs[tid] = hi;
    }
    const double r2 = sum_partials(part_r2, (int)gridDim.x, red_d);
    const double h2 = block_sum(abs2(hi), red_d);
    C arrow = czero(C());
    if (A.kept > 0) arrow = block_sum(tid < A.kept ? bi * hi : czero(C()), red_s);
    __shared__ double nb2;
    __shared__ C coupled;
    if (tid == 0) {
        const double b = r2 - h2;
        nb2 = b;
        coupled = arrow;
        A.ta[k] = alpha;
        if (!A.first) {
            A.tb[k - 1] = bprev;
            A.lg_prev[3] = b2;
        }
        A.sc[0] = 1.0 / sqrt(b);
        A.sc[1] = b;
        A.sc[2] = sqrt(b);
        A.lg[0] = alpha;
        A.lg[1] = r2;
        A.lg[2] = h2;
        *ticket = 0;
    }
    __syncthreads();
    if (tid <= k) {
        const int i = tid;
        C s = ti * hi;
        if (i < A.kept) {
            s = s + bi * hs[A.kept];
        } else {
            if (i > A.kept)
                s = s + bl * hs[i - 1];
            else
                s = s + coupled;
            if (i < k) s = s + bi * hs[i + 1];
        }
        if (kWide && i == k) s = s + as_c(nb2, C());
        A.c[i] = s;
    }
}

template <class T>
using Kern = void (*)(const SweepArgs<T>, long, typename Store<T>::C *, double *, unsigned *);
template <class T>
struct Variant {
    Kern<T> kern;
    size_t smem;
};
template <class T, int NC, int G>
constexpr Variant<T> variant() {
    return Variant<T>{k_sweep<T, NC, G>, Shape<T, NC, G>::kSmem};
}

}  // namespace

template <class T>
int launch_sweep(const SweepArgs<T> &a, Scratch &s, cudaStream_t st) {
    using C = typename Store<T>::C;
    // By groups (1, 2, 4, 8) and columns per group (to 8 or 10, 12, 14, 16).
    static const Variant<T> kern[4][4] = {
        {variant<T, 8, 1>(), variant<T, 12, 1>(), variant<T, 16, 1>(), variant<T, 16, 1>()},
        {variant<T, 10, 2>(), variant<T, 12, 2>(), variant<T, 14, 2>(), variant<T, 16, 2>()},
        {variant<T, 10, 4>(), variant<T, 12, 4>(), variant<T, 14, 4>(), variant<T, 16, 4>()},
        {variant<T, 10, 8>(), variant<T, 12, 8>(), variant<T, 14, 8>(), variant<T, 16, 8>()}};
    // SMs of each device; reading them also lets the kernels use their ring
    // there.  Host threads take turns: none sees a device half set up.
    static std::mutex turn;
    static int sms_of[64] = {};
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    {
        std::lock_guard<std::mutex> hold(turn);
        if (dev < 64) sms = sms_of[dev];
        if (sms == 0) {
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (sms <= 0) sms = 148;
            for (const auto &row : kern)
                for (const auto &v : row)
                    if (cudaFuncSetAttribute(v.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem) !=
                        cudaSuccess) {
                        cudaGetLastError();
                        return -1;
                    }
            if (dev < 64) sms_of[dev] = sms;
        }
    }
    // One block per SM on an equal share of the rows, in whole tiles.
    const long tile = 32 * Store<T>::R;
    const long want = std::min<long>(sms, s.max_blocks);
    long chunk = (a.n_pad + want - 1) / want;
    chunk = (chunk + tile - 1) / tile * tile;
    const int nb = (int)((a.n_pad + chunk - 1) / chunk);
    C *part = static_cast<C *>(s.partials);
    double *part_r2 = reinterpret_cast<double *>(part + (size_t)nb * (a.k + 1));
    int lg = 0;
    while ((kCols << lg) < a.k) ++lg;
    const int per = (a.k + (1 << lg) - 1) >> lg;  // columns per group
    const int nc = lg == 0 ? (per <= 8 ? 0 : (per <= 12 ? 1 : 2)) : (std::max(per, 10) - 9) / 2;
    const Variant<T> &v = kern[lg][nc];
    // Launched while the operator's kernel ends (which lets it at its start;
    // that one itself starts when the sweep before is complete): 64^3 FP64
    // 12.2 -> 11.7 ms a call, 101^3 FP32 17.5 -> 16.9 ms.
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nb);
    cfg.blockDim = dim3(kNT);
    cfg.dynamicSmemBytes = v.smem;
    cfg.stream = st;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, v.kern, a, chunk, part, part_r2, s.tickets + kTicketSweep) == cudaSuccess) return 0;
    cudaGetLastError();
    return -1;
}

template int launch_sweep<double>(const SweepArgs<double> &, Scratch &, cudaStream_t);
template int launch_sweep<float>(const SweepArgs<float> &, Scratch &, cudaStream_t);
template int launch_sweep<zd>(const SweepArgs<zd> &, Scratch &, cudaStream_t);
template int launch_sweep<zf>(const SweepArgs<zf> &, Scratch &, cudaStream_t);

}  // namespace trlb
