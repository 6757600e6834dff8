// The warp-parallel dense routines (kernels/dense_warp.cuh) on the CPU: the 32
// lanes are contexts of their own, each run until it meets the others at a
// __syncwarp() or a shuffle.  Between two meetings the lanes run one after the
// other in the order asked for, which is one of the orders that a GPU may take:
// results that depend on it show a missing __syncwarp().
#include <ucontext.h>

#include <cfloat>
#include <cmath>
#include <cstring>
#include <functional>
#include <vector>

#define __device__
#define __forceinline__ inline
static inline double rsqrt(double v) { return 1.0 / std::sqrt(v); }
static inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }

namespace {

constexpr int kLanes = 32;

struct Warp {
    ucontext_t main, ctx[kLanes];
    std::vector<char> stack[kLanes];
    bool done[kLanes];
    int kind[kLanes];  // what the lane waits in (0: nothing)
    unsigned long long put[kLanes], got[kLanes];
    int now = -1;
    bool mixed = false;  // lanes met in different calls
    std::function<void(int)> body;
} *W = nullptr;

void lane_main() {
    const int l = W->now;
    W->body(l);
    W->done[l] = true;
    W->kind[l] = 0;
    swapcontext(&W->ctx[l], &W->main);
}

// Waits until every lane has called this; returns the lanes' values.
const unsigned long long *meet(int kind, unsigned long long v) {
    const int l = W->now;
    W->put[l] = v;
    W->kind[l] = kind;
    swapcontext(&W->ctx[l], &W->main);
    return W->got;
}

bool run_warp(int order, std::function<void(int)> body) {
    Warp w;
    W = &w;
    w.body = std::move(body);
    for (int l = 0; l < kLanes; ++l) {
        w.stack[l].resize(1 << 18);
        w.done[l] = false;
        getcontext(&w.ctx[l]);
        w.ctx[l].uc_stack.ss_sp = w.stack[l].data();
        w.ctx[l].uc_stack.ss_size = w.stack[l].size();
        w.ctx[l].uc_link = &w.main;
        makecontext(&w.ctx[l], lane_main, 0);
    }
    for (;;) {
        int live = 0;
        for (int q = 0; q < kLanes; ++q) {
            const int l = order == 0 ? q : kLanes - 1 - q;
            if (w.done[l]) continue;
            w.now = l;
            swapcontext(&w.main, &w.ctx[l]);
            live += !w.done[l];
        }
        if (live == 0) break;
        for (int l = 0; l < kLanes; ++l) w.mixed |= w.done[l] || w.kind[l] != w.kind[0];
        if (w.mixed) break;
        memcpy(w.got, w.put, sizeof(w.got));
    }
    W = nullptr;
    return !w.mixed;
}

}  // namespace

static inline void __syncwarp() { meet(1, 0); }
static inline unsigned __ballot_sync(unsigned, bool p) {
    const unsigned long long *v = meet(2, p);
    unsigned r = 0;
    for (int l = 0; l < kLanes; ++l) r |= (unsigned)(v[l] != 0) << l;
    return r;
}
template <class T>
static inline T lane_value(int kind, T v, int from) {
    unsigned long long b = 0;
    memcpy(&b, &v, sizeof(T));
    const unsigned long long *all = meet(kind, b);
    memcpy(&v, &all[from], sizeof(T));
    return v;
}
template <class T>
static inline T __shfl_sync(unsigned, T v, int from) {
    return lane_value(3, v, from);
}
template <class T>
static inline T __shfl_xor_sync(unsigned, T v, int o) {
    return lane_value(4, v, W->now ^ o);
}

using std::fabs;
using std::fma;
using std::hypot;
#include "dense_warp.cuh"

using namespace trlb;

// Lanes in ascending (order 0) or descending order.  Returns 0, the routine's
// error, or -1 where the lanes went separate ways.
extern "C" int warp_get_eval(int order, int nd, int locked, const double *alpha, const double *beta, double *lambda,
                             double *res, int vectors, double *ws) {
    int rc[kLanes] = {};
    const bool ok = run_warp(order, [&](int lane) {
        rc[lane] = warp::get_eval(nd, locked, alpha, beta, lambda, res, vectors != 0, ws, lane);
    });
    for (int l = 1; l < kLanes; ++l)
        if (rc[l] != rc[0]) return -1;
    return ok ? rc[0] : -1;
}

extern "C" int warp_get_tvec_a(int order, int nd, int kept, double *alpha, const double *beta, int nlam,
                               const double *lambda, double *yy, double *ws) {
    int rc[kLanes] = {};
    const bool ok = run_warp(order, [&](int lane) {
        rc[lane] = warp::get_tvec_a(nd, kept, alpha, beta, nlam, lambda, yy, ws, lane);
    });
    for (int l = 1; l < kLanes; ++l)
        if (rc[l] != rc[0]) return -1;
    return ok ? rc[0] : -1;
}

extern "C" long warp_ws_doubles(int nd) { return (long)core::dense_ws_doubles(nd); }
