// Thick-restart Lanczos driver with a device-resident basis.
//
// Control flow follows the reference's trlanczos (SRC/trlcore.c:723-1532)
// and ztrlanczos (SRC/ztrlcore.c:436-1286): same restart decisions, same
// convergence tests, same error codes.  What differs is where the data lives
// and how the vector work is done:
//   * the basis is a pool of padded device columns addressed by a device
//     table of column pointers; restarts write Ritz vectors into free slots
//     and re-point the table instead of copying columns;
//   * the matrix-vector product is either the user's callback (device or
//     host pointers) or a built-in sparse operator fused with the alpha dot;
//   * trl_orth/trl_cgs run as project/update kernel pairs; the first pass of
//     every step applies the three-term recurrence on the fly and is issued
//     before the host has seen alpha (its norm doubles as trl_orth's
//     pre-orthogonalisation norm), so a Lanczos step costs one host sync;
//   * with a built-in operator, runs of steps are issued without waiting for
//     the host's decisions, and for long vectors as single sweeps over the
//     basis (kernels/sweep.cu);
//   * the small projected problem stays on the host in FP64.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <cstdlib>
#include <numeric>
#include <string>
#include <vector>

#include "../kernels/coop.h"
#include "../kernels/lanczos_kernels.h"
#include "../kernels/spmv.h"
#include "../kernels/sweep.h"
#include "dense.h"
#include "comm.h"
#include "engine.h"
#include "hostcopy.h"

namespace trlb {

bool is_device_pointer(const void *p) {
    if (!p) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

std::string pe_filename(const char *prefix, int rank, int npes) {
    int ndig = 1;
    for (int lead = npes; lead > 9; lead /= 10) ++ndig;
    std::string base(prefix ? prefix : "");
    const size_t blank = base.find(' ');
    if (blank != std::string::npos) base.resize(blank);
    char num[32];
    std::snprintf(num, sizeof(num), "%0*d", ndig, rank);
    return base + num;
}

LogOut::LogOut(trl_info *info, const char *mode) {
    if (info->log_fp) {
        fp = static_cast<FILE *>(info->log_fp);
    } else if (info->log_file[0] != '\0') {
        const std::string name = pe_filename(info->log_file, info->my_pe, info->npes);
        FILE *f = std::fopen(name.c_str(), mode);
        if (f) {
            fp = f;
            own = true;
        }
    }
}

LogOut::~LogOut() {
    if (own) std::fclose(fp);
}

trlx_stats &last_stats() {
    static thread_local trlx_stats s;
    return s;
}

// Device workspace kept between solves on the calling thread, so repeated
// solves (benchmark steps, batched or seeded workflows) do not pay for
// allocating and freeing the basis pool every call.  Released by
// trlx_release_workspace() or at thread exit.
struct Workspace {
    void *pool = nullptr;
    size_t pool_bytes = 0;
    void *fbuf = nullptr;
    size_t fbuf_bytes = 0;
    void *small = nullptr;  // coefficients, scalars, Ritz matrix, column table
    size_t small_bytes = 0;
    void *partials = nullptr;
    size_t partial_bytes = 0;
    void *out = nullptr;  // staging of final eigenvectors for host evec
    size_t out_bytes = 0;
    void *refine = nullptr;  // FP64 refinement blocks (32-bit bases)
    size_t refine_bytes = 0;
    unsigned *tickets = nullptr;
    double *h_scal = nullptr;
    double *h_log = nullptr;  // pinned copy of the speculative step log and of a run's start
    size_t h_log_len = 0;
    void *saved = nullptr;  // FP64 working vectors at the start of a run of sweeps (32-bit bases)
    size_t saved_bytes = 0;
    int device = -1;
    ~Workspace() { release(); }
    void release() {
        cudaFree(pool);
        cudaFree(fbuf);
        cudaFree(small);
        cudaFree(partials);
        cudaFree(out);
        cudaFree(refine);
        cudaFree(saved);
        cudaFree(tickets);
        cudaFreeHost(h_scal);
        cudaFreeHost(h_log);
        h_log = nullptr;
        h_log_len = 0;
        pool = fbuf = small = partials = out = refine = saved = nullptr;
        out_bytes = refine_bytes = saved_bytes = 0;
        tickets = nullptr;
        h_scal = nullptr;
        pool_bytes = fbuf_bytes = small_bytes = partial_bytes = 0;
        device = -1;
    }
    // Grows buf to at least `bytes`; returns false on allocation failure.  The
    // vectors kept for runs make way: they only save time.
    bool ensure(void **buf, size_t *have, size_t bytes) {
        if (*have >= bytes && *buf) return true;
        cudaFree(*buf);
        *buf = nullptr;
        *have = 0;
        if (bytes == 0) return true;
        cudaError_t e = cudaMalloc(buf, bytes);
        if (e != cudaSuccess && saved) {
            cudaFree(saved);
            saved = nullptr;
            saved_bytes = 0;
            e = cudaMalloc(buf, bytes);
        }
        if (e != cudaSuccess) {
            cudaGetLastError();
            *buf = nullptr;
            return false;
        }
        *have = bytes;
        return true;
    }
};

Workspace &workspace() {
    static thread_local Workspace w;
    int dev = 0;
    cudaGetDevice(&dev);
    if (w.device != dev) {
        w.release();
        w.device = dev;
    }
    return w;
}

void release_workspace() {
    workspace().release();
    release_staging();
    trim_operator_pools();
}

__global__ void k_zero_padding(char *pool, int nslots, size_t slot_bytes, size_t from_byte) {
    const size_t tail = slot_bytes - from_byte;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)nslots * tail;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t s = i / tail, o = i - s * tail;
        pool[s * slot_bytes + from_byte + o] = 0;
    }
}

Options options_from(const trlx_options *o) {
    Options r;
    if (!o) return r;
    r.basis_bits = o->basis_bits == 32 ? 32 : 64;
    r.seed = o->seed ? o->seed : r.seed;
    r.stream = static_cast<cudaStream_t>(o->stream);
    r.refine = o->refine;
    r.profile = o->profile;
    return r;
}

namespace {

enum Scal { kAlpha = 0, kR2Pre = 1, kH2 = 2, kR2Post = 3, kNorm = 4, kNumScal = 8 };

double now_s() {
    using namespace std::chrono;
    return duration<double>(steady_clock::now().time_since_epoch()).count();
}

#define CK(call)                                                                          \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            std::fprintf(stderr, "TRLAN-B200: CUDA error %s at %s:%d\n",                  \
                         cudaGetErrorString(e_), __FILE__, __LINE__);                     \
            return -1001;                                                                 \
        }                                                                                 \
    } while (0)

template <class T>
struct OpTypes;
template <>
struct OpTypes<double> {
    using Fn = trl_matvec;
    using User = double;
};
template <>
struct OpTypes<float> {
    using Fn = trl_matvec;
    using User = double;
};
template <>
struct OpTypes<zd> {
    using Fn = ztrl_matvec;
    using User = trl_dcomplex;
};
template <>
struct OpTypes<zf> {
    using Fn = ztrl_matvec;
    using User = trl_dcomplex;
};

template <class T>
class Engine {
   public:
    using C = typename Store<T>::C;
    static constexpr bool kComplex = std::is_same<C, zd>::value;
    static constexpr bool kWide = std::is_same<T, C>::value;  // FP64 / c128 storage
    using OpFn = typename OpTypes<T>::Fn;
    using User = typename OpTypes<T>::User;

    Engine(OpFn op, trl_uo uo, trl_info *info, int nrow, int mev, double *eval, User *evec, int lde,
           const Options &opt)
        : op_(op), uo_(uo), info_(info), nrow_(nrow), mev_(mev), eval_(eval), evec_(evec), lde_(lde),
          opt_(opt) {}

    ~Engine() { release(); }

    int setup();
    void run();
    // Residual norms on exit (reference: wrk[0:j1] = |beta|, rest alpha).
    void residual_output(double *out, int count) const {
        for (int i = 0; i < count && i < maxlan_; ++i)
            out[i] = i < final_j1_ ? std::fabs(beta_[i]) : alpha_[i];
    }

   private:
    // ---- device helpers ----
    T *col(int j) const { return pool_ + (size_t)lslot_[j] * n_pad_; }
    C *col64(int j) const {
        if constexpr (kWide)
            return reinterpret_cast<C *>(col(j));
        else
            return nullptr;
    }
    int upload_table();
    int apply_op(const C *x, C *y, bool want_alpha);
    int sync_scalars();
    int orth(int m, bool recur, double beta_prev, int kept);
    int cgs(int m, bool pass_done, double *rnrm, bool *irnd_used);
    int normalize_into(int m, double scale_fixed, bool use_r2);
    void rotate_fp64();
    int initial_guess(int *jnd);
    int restart_ritz(int locked, int jml, int kept, int jnd);
    int final_vectors(int jnd, int kept);
    // Checkpoint file of the reference (trl_write_checkpoint /
    // trl_read_checkpoint, SRC/trlaux.c:780-1014): int nrow, int jnd,
    // jnd alphas, jnd betas, jnd + 1 vectors of nrow values.
    template <class ColFn>
    int write_checkpoint(int jnd, ColFn colptr);
    int read_checkpoint(int nec, int *jnd_out);
    int refine_fp64(int k, double *max_res);
    bool spec_enabled() const;
    // The steps accepted (jnd moves on by them), or an error.
    int spec_segment(int *jnd, int S, int kept);
    // Asked of every beta of a run of single-sweep steps: keeps |r|^2 and
    // r^H A r, formed from unnormalised vectors, far from overflow and
    // underflow.  A solve that meets another goes on without such runs.
    bool scale_off_ = false;
    bool sweep_off_ = false;  // a sweep's launch or memory was refused: the solve goes on without
    bool coop_off_ = false;   // the same of a cooperative run's launch
    static bool in_range(double beta) { return beta > 1e-90 && beta < 1e90; }
    // Steps since the last one that was not taken as runs assume, once a run
    // was cut short by one (INT_MAX before).  A run is at most half as long, so
    // that operators whose steps often need a second pass do not have run after
    // run thrown away.
    int streak_ = INT_MAX;
    void took_steps(int n, bool as_assumed) {
        if (streak_ < INT_MAX) streak_ = !as_assumed ? 0 : streak_ > INT_MAX - n ? INT_MAX : streak_ + n;
    }
    bool sweeps(int jnd) const;
    bool coop_steps(int jnd, int S) const;
    size_t partial_doubles() const { return (size_t)scratch_.max_blocks * (P_ + 2) * 2; }
    int upload_run(int j0, int S, int kept);
    int sweep_steps(int j0, int S, int kept);
    bool accept_step(int jnd, int kept, const double *lg, bool sweep);
    void track_ritz(int nd) {
        for (int i = 0; i < nd; ++i) {
            ritz_min_ = std::min(ritz_min_, lambda_[i]);
            ritz_max_ = std::max(ritz_max_, lambda_[i]);
        }
    }
    void log_progress();
    void release();
    void count_launch(int k = 1) { launches_ += k; }
    // Per-kernel-class timing with CUDA events on st_ (options.profile).
    int pbeg();
    void pend(int id, int cls, double bytes);
    void flush_prof();
    double cs() const { return (double)sizeof(C); }
    double sv() const { return (double)sizeof(T); }

    OpFn op_;
    trl_uo uo_;
    trl_info *info_;
    int nrow_, mev_;
    double *eval_;
    User *evec_;
    int lde_;
    Options opt_;

    // modes
    bool user_dev_ = false;
    const trlx_operator *builtin_ = nullptr;
    // Projection kernel form tuned for the built-in operator and this
    // basis' storage width (0: default).
    int proj_form() const {
        if (!builtin_) return 0;
        return sizeof(T) < sizeof(C) ? builtin_->project_form32 : builtin_->project_form;
    }
    bool host_op_ = false;
    // Block-row solve: sums over the ranks of the communicator stored in
    // info->mpicomp by trlx_init_info_comm (nullptr: one GPU).
    Comm *comm_ = nullptr;
    int gsum(double *d, size_t n) { return comm_ ? comm_->sum_device(d, n, st_) : 0; }
    template <class V>
    int gsum_c(V *d, size_t n) {
        return gsum(reinterpret_cast<double *>(d), n * (sizeof(V) / sizeof(double)));
    }
    // After a projection summed over the ranks, |h|^2 comes from the summed h.
    int project_sums(int m) {
        if (!comm_) return 0;
        if (int e = gsum_c(d_coef_, (size_t)m)) return e;
        if (int e = gsum(d_scal_ + kR2Pre, 1)) return e;
        launch_sumsq(reinterpret_cast<const double *>(d_coef_), (long)m * (long)(sizeof(C) / sizeof(double)),
                     d_scal_ + kH2, st_);
        count_launch();
        return 0;
    }
    uint64_t rank_seed(uint64_t s) const { return s + 0x9E3779B97F4A7C15ull * (uint64_t)(comm_ ? comm_->rank : 0); }

    // device state
    long n_pad_ = 0;
    int P_ = 0, maxlan_ = 0;
    T *pool_ = nullptr;
    std::vector<int> lslot_;
    T **d_cols_ = nullptr;
    std::vector<T *> h_cols_;
    C *fbuf_[3] = {nullptr, nullptr, nullptr};  // FP64 q_cur, q_prev, r (narrow storage)
    C *qa64_ = nullptr, *qb64_ = nullptr, *r64_ = nullptr;
    C *d_coef_ = nullptr;
    double *d_scal_ = nullptr, *h_scal_ = nullptr;
    double *d_Y_ = nullptr;
    double *d_log_ = nullptr, *h_log_ = nullptr;  // speculative steps: alpha, |r|^2 pre/post, |h|^2
    // Single-sweep steps: V^H r (in d_coef_), T h, alphas, betas and scalars,
    // contiguous and before the log, with the pinned copy a run starts from.
    C *d_sc_c_ = nullptr;
    double *d_sc_ta_ = nullptr, *d_sc_tb_ = nullptr, *d_sc_s_ = nullptr, *d_sc_dot_ = nullptr;
    double *h_sweep_ = nullptr;
    size_t sweep_doubles() const { return (2 * sizeof(C) / sizeof(double) + 2) * (size_t)P_ + 8; }
    long long discarded_ = 0;                     // speculative operator applications rerun
    long long spec_accepted_ = 0;
    long long coop_segments_ = 0;
    Scratch scratch_;
    cudaStream_t st_ = nullptr;
    bool own_stream_ = false;
    User *hx_ = nullptr, *hy_ = nullptr;  // pinned staging for host operators
    // Per-step op / orth timing: two sets of (start, after op, after orth)
    // events used alternately; a step's set is read at the next step, after
    // that step's scalar sync has retired it, so timing adds no host wait.
    cudaEvent_t ev_[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};  // [6], [7]: speculative segments
    int evset_ = 0, ev_pending_ = -1;
    void tm_begin() {
        if (ev_pending_ == evset_) tm_collect(true);
        cudaEventRecord(ev_[3 * evset_], st_);
    }
    void tm_mid() { cudaEventRecord(ev_[3 * evset_ + 1], st_); }
    void tm_end() {
        if (ev_pending_ >= 0 && ev_pending_ != evset_) tm_collect(false);
        cudaEventRecord(ev_[3 * evset_ + 2], st_);
        ev_pending_ = evset_;
        evset_ ^= 1;
    }
    void tm_collect(bool wait) {
        if (ev_pending_ < 0) return;
        cudaEvent_t *e = ev_ + 3 * ev_pending_;
        if (wait)
            cudaEventSynchronize(e[2]);
        else if (cudaEventQuery(e[2]) != cudaSuccess)
            return;
        float a = 0, b = 0;
        cudaEventElapsedTime(&a, e[0], e[1]);
        cudaEventElapsedTime(&b, e[1], e[2]);
        t_op_ += a * 1e-3;
        t_orth_ += b * 1e-3;
        ev_pending_ = -1;
    }

    // host state (reference names)
    std::vector<double> alpha_, beta_, alfrot_, betrot_, rot_, lambda_, res_, yy_, wrk2_;
    TridiagVectors tridiag_;
    int final_j1_ = 0;
    double ritz_min_ = 1e300, ritz_max_ = -1e300;  // extreme Ritz values seen (spectrum bounds)
    long long launches_ = 0;
    int syncs_ = 0;
    double t_op_ = 0, t_orth_ = 0, t_res_ = 0;
    double fl_ = 0, fl_h_ = 0, fl_r_ = 0;  // flop counts (excluding matvec)
    double setup_seconds_ = 0;
    struct ProfRec {
        cudaEvent_t a, b;
        int cls;
        double bytes;
    };
    std::vector<ProfRec> prof_;
    std::vector<cudaEvent_t> evpool_;
    size_t evnext_ = 0;
    double kt_[8] = {0}, kb_[8] = {0};
    long long kc_[8] = {0};
};

template <class T>
int Engine<T>::pbeg() {
    if (!opt_.profile) return -1;
    if (evnext_ + 2 > evpool_.size()) {
        for (int k = 0; k < 64; ++k) {
            cudaEvent_t e;
            cudaEventCreate(&e);
            evpool_.push_back(e);
        }
    }
    cudaEvent_t a = evpool_[evnext_++];
    cudaEventRecord(a, st_);
    prof_.push_back(ProfRec{a, nullptr, 0, 0.0});
    return (int)prof_.size() - 1;
}

template <class T>
void Engine<T>::pend(int id, int cls, double bytes) {
    if (id < 0) return;
    cudaEvent_t b = evpool_[evnext_++];
    cudaEventRecord(b, st_);
    prof_[id].b = b;
    prof_[id].cls = cls;
    prof_[id].bytes = bytes;
}

// All recorded events have completed when this runs (after a stream sync).
template <class T>
void Engine<T>::flush_prof() {
    for (auto &r : prof_) {
        if (!r.b) continue;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, r.a, r.b);
        kt_[r.cls] += ms * 1e-3;
        kb_[r.cls] += r.bytes;
        kc_[r.cls] += 1;
    }
    prof_.clear();
    evnext_ = 0;
}

// ---------------------------------------------------------------------------
template <class T>
int Engine<T>::setup() {
    maxlan_ = info_->maxlan;
    n_pad_ = ((long)nrow_ + 255) / 256 * 256;
    P_ = 2 * maxlan_ + 2;
    user_dev_ = is_device_pointer(evec_);
    if constexpr (kComplex) {
        if ((void *)op_ == (void *)&trlx_zmatvec && info_->mvparam) builtin_ = static_cast<trlx_operator *>(info_->mvparam);
    } else {
        if ((void *)op_ == (void *)&trlx_matvec && info_->mvparam) builtin_ = static_cast<trlx_operator *>(info_->mvparam);
    }
    if (builtin_) {
        if (builtin_->nrow != nrow_ || trlb::op_complex(builtin_) != kComplex) {
            std::fprintf(stderr, "TRLAN-B200: built-in operator does not match the problem.\n");
            return -6;
        }
    }
    host_op_ = !builtin_ && !user_dev_;
    if (info_->mpicomp) comm_ = static_cast<trlx_comm *>(info_->mpicomp)->impl;
    if (builtin_ && builtin_->halo && !comm_) {
        std::fprintf(stderr, "TRLAN-B200: distributed operator without a communicator in info.\n");
        return -6;
    }

    if (opt_.stream) {
        st_ = opt_.stream;
    } else {
        CK(cudaStreamCreate(&st_));  // blocking: ordered with legacy-stream user work
        own_stream_ = true;
    }
    const double t_alloc0 = now_s();
    Workspace &ws = workspace();
    const size_t pool_bytes = (size_t)P_ * n_pad_ * sizeof(T);
    if (!ws.ensure(&ws.pool, &ws.pool_bytes, pool_bytes)) {
        ws.release();
        std::fprintf(stderr, "TRLAN-B200: cannot allocate %.2f GB basis pool.\n", pool_bytes / 1e9);
        return -5;
    }
    pool_ = static_cast<T *>(ws.pool);
    // Rows >= nrow of every column must read as zero (kernels run over n_pad).
    {
        const size_t slot = (size_t)n_pad_ * sizeof(T), from = (size_t)nrow_ * sizeof(T);
        if (slot > from) {
            k_zero_padding<<<1024, 256, 0, st_>>>(reinterpret_cast<char *>(pool_), P_, slot, from);
            count_launch();
        }
    }
    lslot_.resize(P_);
    for (int i = 0; i < P_; ++i) lslot_[i] = i;
    h_cols_.resize(P_);
    if (!kWide) {
        if (!ws.ensure(&ws.fbuf, &ws.fbuf_bytes, 3 * sizeof(C) * n_pad_)) return -5;
        for (int k = 0; k < 3; ++k) fbuf_[k] = static_cast<C *>(ws.fbuf) + (size_t)k * n_pad_;
        CK(cudaMemsetAsync(ws.fbuf, 0, 3 * sizeof(C) * n_pad_, st_));
        qa64_ = fbuf_[0];
        qb64_ = fbuf_[1];
        r64_ = fbuf_[2];
    }
    // Small buffers carved from one allocation (256-byte aligned pieces).
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t log_len = 4 * ((size_t)maxlan_ + 2), b_coef = al(sizeof(double) * (sweep_doubles() + log_len)),
                 b_scal = al(sizeof(double) * kNumScal), b_Y = al(sizeof(double) * (size_t)maxlan_ * maxlan_),
                 b_cols = al(sizeof(T *) * P_);
    if (!ws.ensure(&ws.small, &ws.small_bytes, b_coef + b_scal + b_Y + b_cols)) return -5;
    char *sp = static_cast<char *>(ws.small);
    d_coef_ = reinterpret_cast<C *>(sp);
    d_sc_c_ = d_coef_ + P_;
    d_sc_ta_ = reinterpret_cast<double *>(d_sc_c_ + P_);
    d_sc_tb_ = d_sc_ta_ + P_;
    d_sc_s_ = d_sc_tb_ + P_;
    d_sc_dot_ = d_sc_s_ + 4;
    d_log_ = d_sc_s_ + 8;  // read back together with the flag before it
    d_scal_ = reinterpret_cast<double *>(sp + b_coef);
    d_Y_ = reinterpret_cast<double *>(sp + b_coef + b_scal);
    d_cols_ = reinterpret_cast<T **>(sp + b_coef + b_scal + b_Y);
    const size_t host_len = 4 + log_len + sweep_doubles() + log_len;
    if (ws.h_log_len < host_len) {
        cudaFreeHost(ws.h_log);
        ws.h_log = nullptr;
        ws.h_log_len = 0;
        CK(cudaMallocHost(&ws.h_log, sizeof(double) * host_len));
        ws.h_log_len = host_len;
    }
    h_log_ = ws.h_log + 4;
    h_sweep_ = h_log_ + log_len;
    CK(cudaMemsetAsync(d_scal_, 0, sizeof(double) * kNumScal, st_));
    if (!ws.h_scal) CK(cudaMallocHost(&ws.h_scal, sizeof(double) * kNumScal));
    h_scal_ = ws.h_scal;
    scratch_.max_blocks = 148 * 8;
    scratch_.max_cols = P_;
    if (!ws.ensure(&ws.partials, &ws.partial_bytes,
                           (size_t)scratch_.max_blocks * (P_ + 2) * sizeof(zd)))
        return -5;
    scratch_.partials = ws.partials;
    if (!ws.tickets) CK(cudaMalloc(&ws.tickets, sizeof(unsigned) * kNumTickets));
    scratch_.tickets = ws.tickets;
    CK(cudaMemsetAsync(scratch_.tickets, 0, sizeof(unsigned) * kNumTickets, st_));
    setup_seconds_ = now_s() - t_alloc0;
    if (host_op_) {
        CK(cudaMallocHost(&hx_, sizeof(User) * (size_t)nrow_));
        CK(cudaMallocHost(&hy_, sizeof(User) * (size_t)nrow_));
    }
    for (auto &e : ev_) CK(cudaEventCreate(&e));
    size_t mm = (size_t)maxlan_ + 1;
    alpha_.assign(mm, 0.0);
    beta_.assign(mm, 0.0);
    alfrot_.assign(mm, 0.0);
    betrot_.assign(mm, 0.0);
    rot_.assign(mm * mm, 0.0);
    lambda_.assign(mm, 0.0);
    res_.assign(mm, 0.0);
    yy_.assign(mm * mm, 0.0);
    wrk2_.assign(4 * mm, 0.0);
    return upload_table();
}

template <class T>
void Engine<T>::release() {
    // Device buffers belong to the thread's workspace and stay allocated.
    cudaStreamSynchronize(st_);
    cudaFreeHost(hx_);
    cudaFreeHost(hy_);
    hx_ = hy_ = nullptr;
    for (auto e : ev_)
        if (e) cudaEventDestroy(e);
    for (auto e : evpool_) cudaEventDestroy(e);
    if (own_stream_) cudaStreamDestroy(st_);
    pool_ = nullptr;
}

template <class T>
int Engine<T>::upload_table() {
    for (int j = 0; j < P_; ++j) h_cols_[j] = col(j);
    CK(cudaMemcpyAsync(d_cols_, h_cols_.data(), sizeof(T *) * P_, cudaMemcpyHostToDevice, st_));
    // The host vector must stay unchanged until the copy ran.
    CK(cudaStreamSynchronize(st_));
    return 0;
}

template <class T>
int Engine<T>::sync_scalars() {
    CK(cudaMemcpyAsync(h_scal_, d_scal_, sizeof(double) * kNumScal, cudaMemcpyDeviceToHost, st_));
    CK(cudaStreamSynchronize(st_));
    ++syncs_;
    if (!prof_.empty()) flush_prof();
    return 0;
}

// y = A x (+ alpha into d_scal_[kAlpha]).
template <class T>
int Engine<T>::apply_op(const C *x, C *y, bool want_alpha) {
    double *aout = want_alpha ? d_scal_ + kAlpha : nullptr;
    if (builtin_) {
        int pid = pbeg();
        if constexpr (kComplex) {
            spmv_fused_cplx(builtin_, x, y, n_pad_, aout, &scratch_, st_);
        } else {
            const double *xin = x;
            if (builtin_->halo) {
                if (int e = halo_exchange(builtin_, x, st_, &xin)) return e;
                count_launch();
            }
            spmv_fused_real(builtin_, xin, y, n_pad_, aout, &scratch_, st_);
        }
        pend(pid, TRLX_K_SPMV, spmv_bytes(builtin_));
        count_launch();
        if (aout)
            if (int e = gsum(aout, 1)) return e;
    } else if (!host_op_) {
        // The user's operator sees device pointers; our stream is a blocking
        // stream, so work it issues on the legacy default stream is ordered.
        CK(cudaStreamSynchronize(st_));
        op_(nrow_, 1, reinterpret_cast<const User *>(x), (int)n_pad_, reinterpret_cast<User *>(y), (int)n_pad_,
            info_->mvparam);
        // The operator may have used any stream: wait for all of its work.
        CK(cudaDeviceSynchronize());
        if (want_alpha) {
            int pid = pbeg();
            launch_dot<C>(x, y, n_pad_, aout, scratch_, st_);
            pend(pid, TRLX_K_DOT, 2.0 * nrow_ * cs());
            count_launch();
            if (int e = gsum(aout, 1)) return e;
        }
    } else {
        CK(cudaMemcpyAsync(hx_, x, sizeof(User) * nrow_, cudaMemcpyDeviceToHost, st_));
        CK(cudaStreamSynchronize(st_));
        op_(nrow_, 1, hx_, nrow_, hy_, nrow_, info_->mvparam);
        CK(cudaMemcpyAsync(y, hy_, sizeof(User) * nrow_, cudaMemcpyHostToDevice, st_));
        if (want_alpha) {
            int pid = pbeg();
            launch_dot<C>(x, y, n_pad_, aout, scratch_, st_);
            pend(pid, TRLX_K_DOT, 2.0 * nrow_ * cs());
            count_launch();
            if (int e = gsum(aout, 1)) return e;
        }
    }
    info_->matvec++;
    return 0;
}

// Normalise r into basis column m (and the FP64 copy).
template <class T>
int Engine<T>::normalize_into(int m, double scale_fixed, bool use_r2) {
    const double *r2 = use_r2 ? d_scal_ + kNorm : nullptr;
    int pid = pbeg();
    if constexpr (kWide) {
        launch_normalize<T>(r64_, n_pad_, r2, scale_fixed, r64_, nullptr, st_);
    } else {
        launch_normalize<T>(r64_, n_pad_, r2, scale_fixed, r64_, col(m), st_);
    }
    pend(pid, TRLX_K_NORMALIZE, 2.0 * nrow_ * cs() + (kWide ? 0.0 : nrow_ * sv()));
    count_launch();
    return 0;
}

// After column m got its vector: FP64 copies move one step.
template <class T>
void Engine<T>::rotate_fp64() {
    if constexpr (!kWide) {
        C *new_cur = r64_;
        C *old_prev = qb64_;
        qb64_ = qa64_;
        qa64_ = new_cur;
        r64_ = old_prev;
    }
}

// Gram-Schmidt against columns 0..m-1 (reference trl_cgs,
// SRC/trlcore.c:2913-3117).  When pass_done, the first project/update pass
// has already been issued and its scalars are in h_scal_.
template <class T>
int Engine<T>::cgs(int m, bool pass_done, double *rnrm, bool *irnd_used) {
    const int maxorth = 3;
    int irnd = 0;
    double normrr2 = 0.0, normdiff2 = 0.0;
    if (m > 0) {
        int cnt = 0;
        bool first = true;
        while (cnt <= maxorth) {
            if (!(first && pass_done)) {
                Recur<C> none;
                int p1 = pbeg();
                launch_project<T>(d_cols_, m, n_pad_, r64_, none, d_coef_, d_scal_ + kR2Pre, scratch_, st_, proj_form());
                pend(p1, TRLX_K_PROJECT, (double)m * nrow_ * sv() + nrow_ * cs());
                if (int e = project_sums(m)) return e;
                int p2 = pbeg();
                launch_update<T>(d_cols_, m, n_pad_, r64_, none, d_coef_, r64_, d_scal_ + kR2Post, scratch_, st_);
                pend(p2, TRLX_K_UPDATE, (double)m * nrow_ * sv() + 2.0 * nrow_ * cs());
                count_launch(2);
                if (int e = gsum(d_scal_ + kR2Post, 1)) return e;
                if (int e = sync_scalars()) return e;
            }
            first = false;
            double ud = 0.0;
            if (uo_) {
                if constexpr (!kComplex) {
                    if (host_op_) {
                        CK(cudaMemcpy(hx_, r64_, sizeof(double) * nrow_, cudaMemcpyDeviceToHost));
                        uo_(nrow_, hx_, &ud);
                        CK(cudaMemcpy(r64_, hx_, sizeof(double) * nrow_, cudaMemcpyHostToDevice));
                    } else {
                        uo_(nrow_, reinterpret_cast<double *>(r64_), &ud);
                    }
                    launch_dot<C>(r64_, r64_, n_pad_, d_scal_ + kR2Post, scratch_, st_);
                    count_launch();
                    if (int e = gsum(d_scal_ + kR2Post, 1)) return e;
                    if (int e = sync_scalars()) return e;
                }
            }
            info_->north++;
            cnt++;
            normdiff2 = h_scal_[kH2];
            normrr2 = h_scal_[kR2Post];
            if (uo_) normdiff2 += ud * ud;
            *rnrm = std::sqrt(normrr2);
            if (DBL_EPSILON * normrr2 > normdiff2) break;
            if ((cnt > 1 && (m * DBL_EPSILON * DBL_EPSILON * (normrr2 + normdiff2) < normdiff2)) ||
                !(normrr2 > DBL_MIN)) {
                // Linearly dependent on the basis: try one fresh random vector.
                if (irnd > 0) break;
                cnt = 0;
                irnd++;
                info_->nrand++;
                launch_random<C>(r64_, nrow_, n_pad_, rank_seed(opt_.seed + 7919ull * (uint64_t)info_->nrand), st_);
                count_launch();
            }
        }
        if (normrr2 < normdiff2 && !uo_) return -203;
    }
    if (*rnrm > DBL_MIN) {
        normalize_into(m, 1.0 / *rnrm, false);
    } else {
        return -204;
    }
    if (irnd > 0) *rnrm = 0.0;
    if (irnd_used) *irnd_used = irnd > 0;
    return 0;
}

// trl_orth (SRC/trlcore.c:1766-1975): r (in r64_) against columns 0..m-1,
// result normalised into column m; sets alpha_[m-1] (from the device) and
// beta_[m-1].
template <class T>
int Engine<T>::orth(int m, bool recur, double beta_prev, int kept) {
    const int jnd = m, jm1 = jnd - 1;
    // Optimistic first Gram-Schmidt pass (the full pass is taken in almost
    // every step); the recurrence r = y - alpha qa - beta qb is applied on
    // the fly with alpha read from device memory.
    Recur<C> rec;
    if (recur) {
        rec.x = qa64_;
        rec.xp = qb64_;
        rec.alpha = d_scal_ + kAlpha;
        rec.beta = beta_prev;
        rec.on = 1;
    }
    const double recb = recur ? 2.0 * nrow_ * cs() : 0.0;
    int p1 = pbeg();
    launch_project<T>(d_cols_, m, n_pad_, r64_, rec, d_coef_, d_scal_ + kR2Pre, scratch_, st_, proj_form());
    pend(p1, TRLX_K_PROJECT, (double)m * nrow_ * sv() + nrow_ * cs() + recb);
    if (int e = project_sums(m)) return e;
    int p2 = pbeg();
    launch_update<T>(d_cols_, m, n_pad_, r64_, rec, d_coef_, r64_, d_scal_ + kR2Post, scratch_, st_);
    pend(p2, TRLX_K_UPDATE, (double)m * nrow_ * sv() + 2.0 * nrow_ * cs() + recb);
    count_launch(2);
    if (int e = gsum(d_scal_ + kR2Post, 1)) return e;
    if (int e = sync_scalars()) return e;
    alpha_[jnd - 1] = h_scal_[kAlpha];
    const double normrr2 = h_scal_[kR2Pre];
    if (!(normrr2 >= 0.0) || !(normrr2 <= DBL_MAX)) return -102;
    beta_[jnd - 1] = std::sqrt(normrr2);
    double tmp = alpha_[jnd - 1] * alpha_[jnd - 1];
    if (jm1 > kept) {
        tmp += beta_[jm1 - 1] * beta_[jm1 - 1];
        fl_ += 2 * nrow_ + 4;
    } else if (kept > 0) {
        for (int i = 0; i < jm1; ++i) tmp += beta_[i] * beta_[i];
        fl_ += 2 * (nrow_ + kept + 2);
    }
    bool usecgs;
    if (jm1 == kept) {
        usecgs = true;
    } else if (jnd >= info_->ntot) {
        usecgs = false;
    } else if (DBL_EPSILON * normrr2 >= tmp) {
        double anorm = 0.0;
        for (int i = 0; i < jnd; ++i) anorm = std::max(anorm, std::fabs(alpha_[i]) + std::fabs(beta_[i]));
        usecgs = beta_[jm1] < DBL_EPSILON * anorm * info_->ntot;
    } else {
        usecgs = true;
    }
    if (usecgs) {
        const int nr = info_->nrand, no = info_->north;
        double rnrm = beta_[jnd - 1];
        int st = cgs(m, true, &rnrm, nullptr);
        fl_ += 4 * nrow_ * ((info_->north - no) * jnd + info_->nrand - nr) + nrow_;
        if (st) return st;
        beta_[jnd - 1] = rnrm;
    } else {
        // Local re-orthogonalisation against the last one or two vectors:
        // restore the components the optimistic pass removed from the older
        // columns, then apply the reference's local update and scaling.
        std::vector<C> h(m);
        CK(cudaMemcpy(h.data(), d_coef_, sizeof(C) * m, cudaMemcpyDeviceToHost));
        std::vector<C> g(m);
        const int nloc = std::min(2, m);
        for (int c = 0; c < m; ++c) {
            if (c < m - nloc) {
                if constexpr (kComplex)
                    g[c] = zd{-h[c].x, -h[c].y};
                else
                    g[c] = -h[c];
            } else {
                if constexpr (kComplex)
                    g[c] = zd{0.0, 0.0};
                else
                    g[c] = 0.0;
            }
        }
        if (m > nloc) {
            CK(cudaMemcpyAsync(d_coef_, g.data(), sizeof(C) * m, cudaMemcpyHostToDevice, st_));
            Recur<C> none;
            launch_update<T>(d_cols_, m, n_pad_, r64_, none, d_coef_, r64_, d_scal_ + kR2Post, scratch_, st_);
            count_launch();
        }
        double dlast;
        if constexpr (kComplex)
            dlast = h[m - 1].x;
        else
            dlast = h[m - 1];
        alpha_[jnd - 1] += dlast;
        normalize_into(m, 1.0 / beta_[jnd - 1], false);
        fl_ += (jnd > 1 ? 9 : 5) * nrow_;
    }
    if (beta_[jnd - 1] <= DBL_EPSILON * std::fabs(alpha_[jnd - 1]))
        beta_[jnd - 1] = 0.0;
    else if (jnd >= info_->ntot)
        beta_[jnd - 1] = 0.0;
    return 0;
}

// trl_initial_guess (SRC/trlcore.c:1577-1763), without checkpoint reading
// beyond what the caller staged: the start vector is column nec of evec
// (guess == 1), the ones vector (guess == 0), or ones with -guess random
// perturbations (guess < 0).
template <class T>
int Engine<T>::initial_guess(int *jnd_out) {
    const int nec = info_->nec;
    const size_t ue = sizeof(User);
    // Locked vectors 0..nec-1 from the user's evec.
    for (int j = 0; j < nec; ++j) {
        C *dst = kWide ? reinterpret_cast<C *>(col(j)) : r64_;
        CK(user_dev_ ? cudaMemcpyAsync(dst, evec_ + (size_t)j * lde_, ue * nrow_, cudaMemcpyDeviceToDevice, st_)
                     : host_copy(dst, evec_ + (size_t)j * lde_, ue * nrow_, cudaMemcpyHostToDevice, st_));
        if (!kWide) {
            launch_store<T>(r64_, n_pad_, col(j), st_);
            count_launch();
        }
    }
    // Start vector into r64_.
    if constexpr (kWide) r64_ = reinterpret_cast<C *>(col(nec));
    int kept0 = nec;  // vectors before the start vector
    if (info_->guess > 1) {
        if (int e = read_checkpoint(nec, &kept0)) return e;
        if constexpr (kWide) r64_ = reinterpret_cast<C *>(col(kept0));
    } else if (info_->guess == 1) {
        CK(user_dev_ ? cudaMemcpyAsync(r64_, evec_ + (size_t)nec * lde_, ue * nrow_, cudaMemcpyDeviceToDevice, st_)
                     : host_copy(r64_, evec_ + (size_t)nec * lde_, ue * nrow_, cudaMemcpyHostToDevice, st_));
    } else {
        std::vector<User> ones(nrow_);
        for (auto &v : ones) {
            if constexpr (kComplex)
                v = trl_dcomplex{1.0, 0.0};
            else
                v = 1.0;
        }
        const int nran = 2 * (std::max(0, 1 - info_->guess) / 2);
        if (nran > 0 && nran < nrow_) {
            for (int k = 0; k + 1 < nran; k += 2) {
                long idx = (long)(nrow_ * uniform01(opt_.seed, (uint64_t)k));
                double pert = uniform01(opt_.seed, (uint64_t)k + 1) - 0.5;
                if constexpr (kComplex)
                    ones[idx].r += pert;
                else
                    ones[idx] += pert;
            }
            fl_ += nran + nran;
        }
        CK(host_copy(r64_, ones.data(), ue * nrow_, cudaMemcpyHostToDevice, st_));
        if (nran >= nrow_) {
            launch_random<C>(r64_, nrow_, n_pad_, rank_seed(opt_.seed), st_);
            count_launch();
            info_->nrand++;
        }
    }
    launch_dot<C>(r64_, r64_, n_pad_, d_scal_ + kR2Post, scratch_, st_);
    count_launch();
    if (int e = gsum(d_scal_ + kR2Post, 1)) return e;
    if (int e = sync_scalars()) return e;
    double normr2 = h_scal_[kR2Post];
    double rnrm = 0.0;
    if (normr2 >= DBL_MIN && normr2 <= DBL_MAX) {
        rnrm = std::sqrt(normr2);
    } else {
        launch_random<C>(r64_, nrow_, n_pad_, rank_seed(opt_.seed ^ 0xA5A5A5A5ull), st_);
        count_launch();
        info_->nrand++;
        launch_dot<C>(r64_, r64_, n_pad_, d_scal_ + kR2Post, scratch_, st_);
        count_launch();
        if (int e = gsum(d_scal_ + kR2Post, 1)) return e;
        if (int e = sync_scalars()) return e;
        rnrm = std::sqrt(h_scal_[kR2Post]);
    }
    const int nr = info_->nrand, no = info_->north;
    int stt = cgs(kept0, false, &rnrm, nullptr);
    fl_ += 4 * nrow_ * ((info_->north - no) * kept0 + info_->nrand - nr) + nrow_;
    if (stt) return stt;
    if constexpr (!kWide) {
        // FP64 copy of the start vector becomes q_cur.
        rotate_fp64();
    }
    *jnd_out = kept0;
    return 0;
}

// Restart: Ritz vectors of columns locked..jnd-1 with coefficients yy_
// (jml x kept) into free slots, then re-point the table.
template <class T>
int Engine<T>::restart_ritz(int locked, int jml, int kept, int jnd) {
    CK(cudaMemcpyAsync(d_Y_, yy_.data(), sizeof(double) * (size_t)jml * kept, cudaMemcpyHostToDevice, st_));
    // Output slots: logical jnd+1 .. jnd+kept are free.
    int pid = pbeg();
    launch_ritz<T>(d_cols_ + locked, jml, n_pad_, d_Y_, jml, kept, d_cols_ + jnd + 1, st_);
    pend(pid, TRLX_K_RITZ, (double)nrow_ * (jml + kept) * sv());
    count_launch();
    std::vector<int> nl;
    nl.reserve(P_);
    for (int j = 0; j < locked; ++j) nl.push_back(lslot_[j]);
    for (int k = 0; k < kept; ++k) nl.push_back(lslot_[jnd + 1 + k]);
    nl.push_back(lslot_[jnd]);  // residual vector follows the kept ones
    for (int j = locked; j < jnd; ++j) nl.push_back(lslot_[j]);
    for (int j = jnd + 1 + kept; j < P_; ++j) nl.push_back(lslot_[j]);
    lslot_ = nl;
    return upload_table();
}

template <class T>
template <class ColFn>
int Engine<T>::write_checkpoint(int jnd, ColFn colptr) {
    const std::string name = pe_filename(info_->cpfile, info_->my_pe, info_->npes);
    FILE *fp = std::fopen(name.c_str(), "wb");
    if (!fp) {
        std::printf("TRL_WRITE_CHECKPOINT: failed to open file: %s.\n", name.c_str());
        return -221;
    }
    auto fail = [&](int code) {
        std::fclose(fp);
        return code;
    };
    const int nrow = nrow_;
    if (std::fwrite(&nrow, sizeof(int), 1, fp) != 1 || std::fwrite(&jnd, sizeof(int), 1, fp) != 1) return fail(-222);
    if (jnd > 0 && (std::fwrite(alpha_.data(), sizeof(double), jnd, fp) != (size_t)jnd ||
                    std::fwrite(beta_.data(), sizeof(double), jnd, fp) != (size_t)jnd))
        return fail(-222);
    std::vector<User> h(nrow_);
    for (int i = 0; i <= jnd; ++i) {
        const C *src = colptr(i);
        if (host_copy(h.data(), src, sizeof(User) * nrow_, cudaMemcpyDeviceToHost, st_) != cudaSuccess)
            return fail(-1001);
        if (std::fwrite(h.data(), sizeof(User), nrow_, fp) != (size_t)nrow_) return fail(-222);
    }
    if (std::fclose(fp) != 0) return -223;
    info_->wrds_out += jnd * (nrow_ + nrow_ + 2) + nrow_ + 2;
    return 0;
}

// Restart from a checkpoint (guess > 1): kept vectors into columns
// nec..nec+jf-1 with their alpha/beta, the last vector of the file becomes
// the start vector, orthogonalised against the kept ones.  All jf + 1
// vectors are read whatever mev is (the reference skips the last one when
// jf >= mev).
template <class T>
int Engine<T>::read_checkpoint(int nec, int *jnd_out) {
    const char *prefix = std::strlen(info_->oldcpf) > 0 ? info_->oldcpf : info_->cpfile;
    const std::string name = pe_filename(prefix, info_->my_pe, info_->npes);
    FILE *fp = std::fopen(name.c_str(), "rb");
    if (!fp) {
        std::printf("TRL_READ_CHECKPOINT: failed to open check-point file %s.\n", name.c_str());
        return -212;
    }
    auto fail = [&](int code) {
        std::fclose(fp);
        return code;
    };
    int nr = 0, jf = 0;
    if (std::fread(&nr, sizeof(int), 1, fp) != 1 || std::fread(&jf, sizeof(int), 1, fp) != 1) return fail(-215);
    if (nr != nrow_) {
        std::printf("TRL_READ_CHECKPOINT: Nrow mismatch.\n");
        return fail(-213);
    }
    if (jf < 0 || nec + jf + 1 > maxlan_) {
        std::printf("TRL_READ_CHECKPOINT: MAXLAN too small.");
        return fail(-214);
    }
    if (jf > 0 && (std::fread(&alpha_[nec], sizeof(double), jf, fp) != (size_t)jf ||
                   std::fread(&beta_[nec], sizeof(double), jf, fp) != (size_t)jf))
        return fail(-215);
    std::vector<User> h(nrow_);
    for (int i = 0; i <= jf; ++i) {
        if (std::fread(h.data(), sizeof(User), nrow_, fp) != (size_t)nrow_) return fail(-215);
        C *dst = kWide ? reinterpret_cast<C *>(col(nec + i)) : r64_;
        CK(host_copy(dst, h.data(), sizeof(User) * nrow_, cudaMemcpyHostToDevice, st_));
        if (!kWide && i < jf) {
            launch_store<T>(r64_, n_pad_, col(nec + i), st_);
            count_launch();
        }
        CK(cudaStreamSynchronize(st_));
    }
    std::fclose(fp);
    info_->wrds_in = jf * (nrow_ + nrow_ + 2) + nrow_ + 2;
    *jnd_out = nec + jf;
    return 0;
}

// Final Ritz vectors (columns 0..jnd-1, yy_ jnd x kept) straight into the
// user's evec (FP64), plus the last Lanczos vector in column kept.
template <class T>
int Engine<T>::final_vectors(int jnd, int kept) {
    CK(cudaMemcpyAsync(d_Y_, yy_.data(), sizeof(double) * (size_t)jnd * kept, cudaMemcpyHostToDevice, st_));
    C *out = nullptr;
    long ldo = lde_;
    C *tmp = nullptr;
    if (user_dev_) {
        out = reinterpret_cast<C *>(evec_);
    } else {
        Workspace &ws = workspace();
        if (!ws.ensure(&ws.out, &ws.out_bytes, sizeof(C) * (size_t)n_pad_ * std::max(kept, 1))) return -5;
        tmp = static_cast<C *>(ws.out);
        out = tmp;
        ldo = n_pad_;
    }
    int pid = pbeg();
    launch_ritz_out<T>(d_cols_, jnd, n_pad_, d_Y_, jnd, kept, out, ldo, nrow_, st_);
    pend(pid, TRLX_K_RITZ, (double)nrow_ * jnd * sv() + (double)nrow_ * kept * cs());
    count_launch();
    const size_t ue = sizeof(User);
    if (!user_dev_ && kept > 0) {
        CK(host_copy_2d(evec_, ue * lde_, tmp, ue * n_pad_, ue * nrow_, kept, cudaMemcpyDeviceToHost, st_));
    }
    // Last Lanczos vector (FP64) into column kept.
    const C *last = kWide ? reinterpret_cast<const C *>(col(jnd)) : qa64_;
    if (kept < mev_) {
        CK(user_dev_ ? cudaMemcpyAsync(evec_ + (size_t)kept * lde_, last, ue * nrow_, cudaMemcpyDeviceToDevice, st_)
                     : host_copy(evec_ + (size_t)kept * lde_, last, ue * nrow_, cudaMemcpyDeviceToHost, st_));
    }
    CK(cudaStreamSynchronize(st_));
    if (info_->cpflag > 0) {
        // Final state: the Ritz vectors and the last Lanczos vector.
        return write_checkpoint(kept, [&](int i) -> const C * {
            if (i == kept) return last;
            return user_dev_ ? reinterpret_cast<const C *>(evec_) + (size_t)i * lde_ : tmp + (size_t)i * n_pad_;
        });
    }
    return 0;
}

// ---- speculative regular steps ---------------------------------------------
// For short vectors the host round trip of every Lanczos step (read alpha
// and the norms, take trl_orth's decisions, launch the next step) costs more
// than the step's kernels, and for long ones it is still 1-2% of a step.
// With a built-in operator the engine issues a run of steps without waiting,
// each assuming the outcome trl_orth takes in almost every step: the full
// classical Gram-Schmidt path with one pass (its stop test passes) and a beta
// that is neither negligible nor a random restart.  Each step logs alpha,
// |r|^2 before and after the pass and |h|^2; the recurrence of the next step
// takes beta = sqrt(|r|^2 after) from that log on the device, and the
// normalisation uses the same value.  The host then replays trl_orth's
// decisions on the logged values in order; the first step whose decisions
// differ and everything after it are discarded (their operator applications
// are subtracted from matvec) and rerun by the sequential path.
// TRLX_SPECULATE=0 disables it.
//
// A run's steps are one cooperative kernel where that is the better one
// (coop_pays) and applies, else single sweeps (sweep.h), else the discrete
// kernels: FP64/c128 bases beyond the columns a sweep takes, and short
// operators that the cooperative kernel does not take.  An accepted step of
// the discrete kernels is bitwise the sequential one; sweeps and the
// cooperative kernel differ from it in rounding only.
// Measured at 2^18 rows, 128 columns: 25.1 ms a solve with the discrete
// kernels, 11.7 with sweeps.
template <class T>
bool Engine<T>::spec_enabled() const {
    if (!builtin_ || uo_ || comm_ || builtin_->halo) return false;
    const char *e = std::getenv("TRLX_SPECULATE");
    return !(e && e[0] == '0');
}

// Whether the speculative steps from basis size jnd on run as single sweeps
// (sweep.h).
template <class T>
bool Engine<T>::sweeps(int jnd) const {
    // A 32-bit basis has no other speculative steps.
    if ((kWide && coop_pays<C>(builtin_, n_pad_)) || jnd < 1 || jnd + 1 > kSweepCols || scale_off_ || sweep_off_)
        return false;
    if ((size_t)P_ * n_pad_ * sizeof(T) > (1ull << 36)) return false;  // 32-bit column offsets, 16-byte units
    const char *e = std::getenv("TRLX_SWEEP");
    return !(e && e[0] == '0');
}

// Whether S of them run in the cooperative kernel (coop.h).
template <class T>
bool Engine<T>::coop_steps(int jnd, int S) const {
    if constexpr (kWide) {
        if (jnd < 1 || !coop_pays<C>(builtin_, n_pad_) || scale_off_ || coop_off_) return false;
        const char *e = std::getenv("TRLX_COOP");
        return !(e && e[0] == '0') && coop_applies<C>(builtin_, n_pad_, jnd + S, partial_doubles());
    }
    return false;
}

template <class T>
bool Engine<T>::accept_step(int jnd, int kept, const double *lg, bool sweep) {
    const int jm1 = jnd - 1;
    const double alpha = lg[0], normrr2 = lg[1], normdiff2 = lg[2], r2post = lg[3];
    if (!(normrr2 >= 0.0) || !(normrr2 <= DBL_MAX)) return false;
    const double beta_pre = std::sqrt(normrr2);
    double tmp = alpha * alpha, fo = 0.0;
    if (jm1 > kept) {
        tmp += beta_[jm1 - 1] * beta_[jm1 - 1];
        fo = 2 * nrow_ + 4;
    } else if (kept > 0) {
        for (int i = 0; i < jm1; ++i) tmp += beta_[i] * beta_[i];
        fo = 2 * (nrow_ + kept + 2);
    }
    bool usecgs;
    if (jm1 == kept) {
        usecgs = true;
    } else if (jnd >= info_->ntot) {
        usecgs = false;
    } else if (DBL_EPSILON * normrr2 >= tmp) {
        double anorm = 0.0;
        for (int i = 0; i < jm1; ++i) anorm = std::max(anorm, std::fabs(alpha_[i]) + std::fabs(beta_[i]));
        anorm = std::max(anorm, std::fabs(alpha) + std::fabs(beta_pre));
        usecgs = beta_pre < DBL_EPSILON * anorm * info_->ntot;
    } else {
        usecgs = true;
    }
    if (!usecgs) return false;
    if (!(DBL_EPSILON * r2post > normdiff2)) return false;  // a second pass would follow
    const double rnrm = std::sqrt(r2post);
    if (!(rnrm > DBL_MIN)) return false;
    if (rnrm <= DBL_EPSILON * std::fabs(alpha) || jnd >= info_->ntot) return false;
    if (sweep && !in_range(rnrm)) {
        scale_off_ = true;
        return false;
    }
    alpha_[jnd - 1] = alpha;
    beta_[jnd - 1] = rnrm;
    alfrot_[jnd - 1] = alpha;
    betrot_[jnd - 1] = rnrm;
    fl_ += jm1 == kept ? 2.0 * jnd * nrow_ + 2.0 * nrow_ : 6.0 * nrow_;
    const double f1 = fl_;
    fl_ += fo + 4.0 * nrow_ * jnd + nrow_;
    fl_h_ += fl_ - f1;
    info_->north++;
    return true;
}

// What a run of S single-sweep steps from basis size j0 starts from: T, the
// first product's coefficients (it is of a finished vector: nothing to
// correct, scale 1), and a log without numbers, which accept_step takes no
// step from: an entry that no kernel writes is not read as one of an earlier
// run.
template <class T>
int Engine<T>::upload_run(int j0, int S, int kept) {
    std::memset(h_sweep_, 0, sizeof(double) * sweep_doubles());
    const size_t log = 4 * ((size_t)S + 1);
    std::fill_n(h_sweep_ + sweep_doubles(), log, std::nan(""));
    double *hc = h_sweep_ + (sizeof(C) / sizeof(double)) * (size_t)P_;
    double *hta = hc + (sizeof(C) / sizeof(double)) * (size_t)P_, *htb = hta + P_, *hs = htb + P_;
    // The step after a restart (j0 == kept) has the arrowhead row for its
    // recurrence, the others the column before (32-bit storage: from its
    // FP64 copy, with the scalar below).
    const size_t cw = sizeof(C) / sizeof(double);
    if (j0 == kept)
        for (int i = 0; i < j0; ++i) hc[cw * i] = beta_[i];
    else if (kWide)
        hc[cw * (size_t)(j0 - 1)] = beta_[j0 - 1];
    for (int i = 0; i < j0; ++i) {
        hta[i] = alpha_[i];
        htb[i] = beta_[i];
    }
    hs[0] = hs[1] = 1.0;
    hs[2] = j0 == kept ? 0.0 : beta_[j0 - 1];
    CK(cudaMemcpyAsync(d_coef_, h_sweep_, sizeof(double) * (sweep_doubles() + log), cudaMemcpyHostToDevice, st_));
    return 0;
}

// Issues S single-sweep steps from basis size j0 (sweep.h): per step one
// product with the vector before its update, and one sweep that finishes
// that vector and projects the next; then the last vector's update and
// normalisation.  The steps log what the discrete kernels log.
template <class T>
int Engine<T>::sweep_steps(int j0, int S, int kept) {
    if (int e = upload_run(j0, S, kept)) return e;
    for (int s = 1; s <= S; ++s) {
        const int k = j0 + s - 1;
        SweepArgs<T> w;
        if constexpr (kWide) {
            w.x = reinterpret_cast<C *>(col(k));
            w.y = reinterpret_cast<C *>(col(k + 1));
        } else {
            w.x = qa64_;
            w.xp = qb64_;
            w.y = r64_;
        }
        int pid = pbeg();
        if constexpr (kComplex)
            spmv_fused_cplx(builtin_, w.x, w.y, n_pad_, d_sc_dot_, &scratch_, st_);
        else
            spmv_fused_real(builtin_, w.x, w.y, n_pad_, d_sc_dot_, &scratch_, st_);
        pend(pid, TRLX_K_SPMV, spmv_bytes(builtin_));
        w.cols = d_cols_;
        w.pool = pool_;
        w.k = k;
        w.kept = kept;
        w.first = s == 1;
        w.n_pad = n_pad_;
        w.dot = d_sc_dot_;
        w.a = d_coef_;
        w.c = d_sc_c_;
        w.ta = d_sc_ta_;
        w.tb = d_sc_tb_;
        w.sc = d_sc_s_;
        w.lg = d_log_ + 4 * (size_t)s;
        w.lg_prev = w.lg - 4;
        pid = pbeg();
        if (int e = launch_sweep<T>(w, scratch_, st_)) return e;
        pend(pid, TRLX_K_PROJECT,
             (double)nrow_ * (k * sv() + (s == 1 ? 3.0 : 4.0) * cs() + (kWide ? 0.0 : cs() + sv())));
        rotate_fp64();
        count_launch(2);
    }
    const int m = j0 + S;
    C *r = kWide ? reinterpret_cast<C *>(col(m)) : qa64_;
    double *r2 = d_log_ + 4 * (size_t)S + 3;
    Recur<C> none;
    int pid = pbeg();
    launch_update<T>(d_cols_, m, n_pad_, r, none, d_coef_, r, r2, scratch_, st_);
    pend(pid, TRLX_K_UPDATE, (double)m * nrow_ * sv() + 2.0 * nrow_ * cs());
    pid = pbeg();
    launch_normalize<T>(r, n_pad_, r2, 0.0, r, kWide ? nullptr : col(m), st_);
    pend(pid, TRLX_K_NORMALIZE, 2.0 * nrow_ * cs() + (kWide ? 0.0 : nrow_ * sv()));
    count_launch(2);
    return 0;
}

template <class T>
int Engine<T>::spec_segment(int *jnd_io, int S, int kept) {
    const int j0 = *jnd_io;
    cudaEventRecord(ev_[6], st_);
    bool done = false, sweep = false, coop = false;
    // Short vectors: the whole run in one cooperative kernel.
    if constexpr (kWide) {
        if (coop_steps(j0, S)) {
            if (upload_run(j0, S, kept)) return -1001;
            // TRLX_COOP_POLLS shortens the grid barrier's wait (to test what follows).
            const char *e = std::getenv("TRLX_COOP_POLLS");
            const long polls = e ? std::max(0L, std::min(kCoopPolls, std::strtol(e, nullptr, 10))) : kCoopPolls;
            int pid = pbeg();
            const int rc = launch_coop<C>(builtin_, reinterpret_cast<C *const *>(d_cols_),
                                          reinterpret_cast<C *>(col(maxlan_ + 1)),
                                          reinterpret_cast<C *>(col(maxlan_ + 2)), n_pad_, j0, S, kept, d_sc_ta_,
                                          d_sc_tb_, d_log_, d_sc_dot_, static_cast<double *>(scratch_.partials),
                                          partial_doubles(), scratch_.tickets + 5, polls, st_);
            if (rc == 0) {
                double bytes = 0.0;
                for (int s = 1; s <= S; ++s) bytes += spmv_bytes(builtin_) + ((double)(j0 + s) + 4.0) * nrow_ * cs();
                pend(pid, TRLX_K_OTHER, bytes);
                info_->matvec += S;
                count_launch();
                coop_segments_++;
                done = coop = true;
            } else {
                coop_off_ = true;
            }
        }
    }
    // The FP64 working vectors of a 32-bit basis at the run's start, which a
    // rejected step or a run that was not issued goes back to.
    const size_t vec = sizeof(C) * n_pad_;
    auto go_back = [&]() -> int {
        Workspace &ws = workspace();
        CK(cudaMemcpyAsync(qa64_, ws.saved, vec, cudaMemcpyDeviceToDevice, st_));
        CK(cudaMemcpyAsync(qb64_, static_cast<char *>(ws.saved) + vec, vec, cudaMemcpyDeviceToDevice, st_));
        return 0;
    };
    if (!done && sweeps(j0)) {
        if constexpr (!kWide) {
            Workspace &ws = workspace();
            if (!ws.ensure(&ws.saved, &ws.saved_bytes, 2 * vec)) {
                sweep_off_ = true;  // no memory for them: steps one by one
                return 0;
            }
            CK(cudaMemcpyAsync(ws.saved, qa64_, vec, cudaMemcpyDeviceToDevice, st_));
            CK(cudaMemcpyAsync(static_cast<char *>(ws.saved) + vec, qb64_, vec, cudaMemcpyDeviceToDevice, st_));
        }
        const int rc = sweep_steps(j0, S, kept);
        if (rc == -1001) return rc;
        if (rc == 0) {
            info_->matvec += S;
            done = sweep = true;
        } else {
            sweep_off_ = true;
            if constexpr (!kWide)
                if (int e = go_back()) return e;
        }
    }
    // The discrete steps know the three-term recurrence only, not the
    // arrowhead row of the step after a restart.
    if (!done && j0 == kept) return 0;
    if constexpr (kWide) {
        for (int s = 1; s <= S && !done; ++s) {
            const int j = j0 + s;
            C *qa = reinterpret_cast<C *>(col(j - 1)), *qb = reinterpret_cast<C *>(col(j - 2)),
              *r = reinterpret_cast<C *>(col(j));
            double *lg = d_log_ + 4 * (size_t)s;
            int pid = pbeg();
            if constexpr (kComplex)
                spmv_fused_cplx(builtin_, qa, r, n_pad_, lg, &scratch_, st_);
            else
                spmv_fused_real(builtin_, qa, r, n_pad_, lg, &scratch_, st_);
            pend(pid, TRLX_K_SPMV, spmv_bytes(builtin_));
            info_->matvec++;
            Recur<C> rec;
            rec.x = qa;
            rec.xp = qb;
            rec.alpha = lg;
            rec.on = 1;
            if (s == 1)
                rec.beta = beta_[j - 2];
            else
                rec.beta_r2 = lg - 4 + 3;
            const double recb = 2.0 * nrow_ * cs();
            int p1 = pbeg();
            launch_project<T>(d_cols_, j, n_pad_, r, rec, d_coef_, lg + 1, scratch_, st_, proj_form());
            pend(p1, TRLX_K_PROJECT, (double)j * nrow_ * sv() + nrow_ * cs() + recb);
            int p2 = pbeg();
            launch_update<T>(d_cols_, j, n_pad_, r, rec, d_coef_, r, lg + 3, scratch_, st_);
            pend(p2, TRLX_K_UPDATE, (double)j * nrow_ * sv() + 2.0 * nrow_ * cs() + recb);
            int p3 = pbeg();
            launch_normalize<T>(r, n_pad_, lg + 3, 0.0, r, nullptr, st_);
            pend(p3, TRLX_K_NORMALIZE, 2.0 * nrow_ * cs());
            count_launch(4);
        }
    } else if (!done) {
        return 0;
    }
    cudaEventRecord(ev_[7], st_);
    // With the four doubles before the log: the cooperative kernel's flag.
    CK(cudaMemcpyAsync(h_log_ - 4, d_log_ - 4, sizeof(double) * (4 * S + 8), cudaMemcpyDeviceToHost, st_));
    CK(cudaStreamSynchronize(st_));
    ++syncs_;
    if (!prof_.empty()) flush_prof();
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev_[6], ev_[7]);
    t_orth_ += ms * 1e-3;
    int acc = 0;
    if (!(coop && h_log_[-4] != 0.0))
        while (acc < S && accept_step(j0 + acc + 1, kept, h_log_ + 4 * (acc + 1), sweep || coop)) ++acc;
    const int dropped = S - acc;
    if (dropped)
        streak_ = 0;
    else
        took_steps(S, true);
    spec_accepted_ += acc;
    info_->matvec -= dropped;
    discarded_ += dropped;
    if constexpr (!kWide) {
        if (dropped) {
            // The working vectors moved on: back to the run's start, and the
            // accepted steps again (the same kernels on the same values).
            if (int e = go_back()) return e;
            if (acc > 0 && sweep_steps(j0, acc, kept)) return -1001;
            discarded_ += acc;
            CK(cudaStreamSynchronize(st_));
            ++syncs_;
            if (!prof_.empty()) flush_prof();
        }
    }
    *jnd_io = j0 + acc;
    return acc;
}

// FP64 refinement of the k converged pairs.  The converged Ritz vectors of a
// 32-bit basis carry the basis' rounding noise, which is spread over the
// whole spectrum; most of its residual comes from the far end.  Each vector
// is passed through a scaled Chebyshev filter of degree kChebDegree that
// damps [a, b] (a = the far end of the wanted Ritz values + 10% of the
// distance to the far spectrum bound, b = that bound, both from the Ritz
// values seen during the solve), then a Rayleigh-Ritz projection in FP64
// over the filtered block (Hermitian for complex problems) gives the pairs
// and their true residuals |A x - theta x|.  Repeated (at most
// kRefinePasses times) until every residual is <= tol * anrm.  Operator
// applications are counted in info->matvec.
template <class T>
int Engine<T>::refine_fp64(int k, double *max_res) {
    using HC = std::conditional_t<kComplex, std::complex<double>, double>;
    static_assert(sizeof(HC) == sizeof(C), "host and device scalar layouts must agree");
    constexpr int kChebDegree = 8;
    constexpr int kRefinePasses = 3;
    trl_info *info = info_;
    if (k <= 0 || !(ritz_max_ > ritz_min_)) return 0;
    const bool low = info->lohi < 0;
    double th_lo = eval_[0], th_hi = eval_[0];
    for (int i = 1; i < k; ++i) {
        th_lo = std::min(th_lo, eval_[i]);
        th_hi = std::max(th_hi, eval_[i]);
    }
    double a, b, ref;
    if (low) {
        const double top = ritz_max_ + 0.01 * (ritz_max_ - th_lo);
        a = th_hi + 0.1 * (top - th_hi);
        b = top;
        ref = th_lo;
    } else {
        const double bot = ritz_min_ - 0.01 * (th_hi - ritz_min_);
        a = bot;
        b = th_lo - 0.1 * (th_lo - bot);
        ref = th_hi;
    }
    if (!(b > a)) return 0;
    const double e = 0.5 * (b - a), c = 0.5 * (b + a);
    const double sigma1 = e / (ref - c);

    Workspace &ws = workspace();
    const size_t vec = (size_t)n_pad_;
    const size_t kk = (size_t)k * k;
    // Blocks W, AW, four work vectors (Chebyshev pair, operator output, zero),
    // then G, H, the combination coefficients, the residual coefficients,
    // |r|^2, a scalar pair and 3k column pointers (all in units of C).
    const size_t elems = (2 * (size_t)k + 4) * vec + 2 * kk + 2 * kk + (size_t)k + 8 + 3 * (size_t)k;
    if (!ws.ensure(&ws.refine, &ws.refine_bytes, elems * sizeof(C))) return -5;
    C *base = static_cast<C *>(ws.refine);
    CK(cudaMemsetAsync(base, 0, elems * sizeof(C), st_));
    C *Wb = base, *AWb = Wb + k * vec, *y0 = AWb + k * vec, *y1 = y0 + vec, *ay = y1 + vec, *zero = ay + vec;
    C *dG = zero + vec, *dH = dG + kk, *dh = dH + kk;
    double *dr2 = reinterpret_cast<double *>(dh + 2 * kk), *dout2 = dr2 + k;
    C **tabW = reinterpret_cast<C **>(dout2 + 8);
    C **tabAWW = tabW + k;
    std::vector<C *> htab(3 * (size_t)k);
    for (int j = 0; j < k; ++j) {
        htab[j] = Wb + j * vec;
        htab[k + j] = AWb + j * vec;
        htab[2 * k + j] = Wb + j * vec;
    }
    CK(cudaMemcpyAsync(tabW, htab.data(), sizeof(C *) * 3 * k, cudaMemcpyHostToDevice, st_));
    // Converged vectors: the caller's device evec or the host staging.
    C *X = user_dev_ ? reinterpret_cast<C *>(evec_) : static_cast<C *>(workspace().out);
    const long ldx = user_dev_ ? lde_ : n_pad_;
    CK(cudaMemcpy2DAsync(Wb, vec * sizeof(C), X, ldx * sizeof(C), nrow_ * sizeof(C), k, cudaMemcpyDeviceToDevice,
                         st_));
    const double tol_abs = info->tol * std::max(info->anrm, 1e-300);
    std::vector<HC> G(kk), H(kk), hv(2 * kk);
    std::vector<double> r2(k), th(k), gl(k);
    std::vector<int> perm(k);
    std::iota(perm.begin(), perm.end(), 0);
    std::stable_sort(perm.begin(), perm.end(), [&](int i, int j) { return eval_[i] < eval_[j]; });
    auto cj = [](const HC &v) {
        if constexpr (kComplex)
            return std::conj(v);
        else
            return v;
    };
    // Symmetric/Hermitian eigen-decomposition of M (k x k) into (w, Z).
    auto eig = [&](std::vector<HC> &M, std::vector<double> &w, std::vector<HC> &Z) -> int {
        if constexpr (kComplex) {
            Z.assign(kk, HC(0.0));
            return herm_eig(k, M.data(), k, w.data(), Z.data(), k);
        } else {
            Z = M;
            return sym_eig(k, Z.data(), k, w.data());
        }
    };
    double worst = -1.0;
    bool refined = false;
    for (int pass = 0; pass < kRefinePasses; ++pass) {
        for (int j = 0; j < k; ++j) {
            C *w = Wb + j * vec;
            // Scaled Chebyshev filter (Zhou & Saad): the wanted end keeps
            // magnitude ~1, [a, b] is damped by ~1/T_d.
            int rc = apply_op(w, ay, false);
            if (rc) return rc;
            launch_cheb(ay, w, nullptr, n_pad_, sigma1 / e, c, 0.0, y1, st_);
            const C *prev = w;
            C *cur = y1, *spare = y0;
            double s1 = sigma1;
            for (int t = 2; t <= kChebDegree; ++t) {
                const double s2 = 1.0 / (2.0 / sigma1 - s1);
                if ((rc = apply_op(cur, ay, false))) return rc;
                C *out = prev == w ? spare : const_cast<C *>(prev);
                launch_cheb(ay, cur, prev, n_pad_, 2.0 * s2 / e, c, -s1 * s2, out, st_);
                prev = cur;
                cur = out;
                s1 = s2;
            }
            CK(cudaMemcpyAsync(w, cur, vec * sizeof(C), cudaMemcpyDeviceToDevice, st_));
            if ((rc = apply_op(w, AWb + j * vec, false))) return rc;
            count_launch(kChebDegree);
        }
        // Columns of W^H W and W^H A W.
        for (int j = 0; j < k; ++j) {
            launch_project<C>(tabW, k, n_pad_, Wb + j * vec, Recur<C>{}, dG + (size_t)j * k, dout2, scratch_, st_);
            launch_project<C>(tabW, k, n_pad_, AWb + j * vec, Recur<C>{}, dH + (size_t)j * k, dout2, scratch_, st_);
        }
        count_launch(2 * k);
        if (int e = gsum_c(dG, kk)) return e;
        if (int e = gsum_c(dH, kk)) return e;
        CK(cudaMemcpyAsync(G.data(), dG, sizeof(C) * kk, cudaMemcpyDeviceToHost, st_));
        CK(cudaMemcpyAsync(H.data(), dH, sizeof(C) * kk, cudaMemcpyDeviceToHost, st_));
        CK(cudaStreamSynchronize(st_));
        ++syncs_;
        for (int i = 0; i < k; ++i)
            for (int j = 0; j <= i; ++j) {
                G[i + j * k] = 0.5 * (G[i + j * k] + cj(G[j + i * k]));
                G[j + i * k] = cj(G[i + j * k]);
                H[i + j * k] = 0.5 * (H[i + j * k] + cj(H[j + i * k]));
                H[j + i * k] = cj(H[i + j * k]);
            }
        // G = Q diag(g) Q^H; B = Q g^{-1/2}; (B^H H B) Z = Z diag(theta).  A
        // filtered block that lost rank keeps the pairs of the last completed
        // pass (or the unrefined ones).
        std::vector<HC> Q, Z, B(kk), P(kk), HB(kk);
        if (eig(G, gl, Q) || !(gl[0] > 1e-14 * gl[k - 1])) break;
        for (int cc = 0; cc < k; ++cc)
            for (int i = 0; i < k; ++i) B[i + cc * k] = Q[i + cc * k] / std::sqrt(gl[cc]);
        for (int cc = 0; cc < k; ++cc)
            for (int i = 0; i < k; ++i) {
                HC acc = 0.0;
                for (int j = 0; j < k; ++j) acc += H[i + j * k] * B[j + cc * k];
                HB[i + cc * k] = acc;
            }
        for (int i = 0; i < k; ++i)
            for (int cc = 0; cc <= i; ++cc) {
                HC acc = 0.0;
                for (int j = 0; j < k; ++j) acc += cj(B[j + i * k]) * HB[j + cc * k];
                P[i + cc * k] = acc;
                P[cc + i * k] = cj(acc);
            }
        if (eig(P, th, Z)) break;
        // Coefficients of the refined vectors, placed so that the i-th
        // smallest refined value lands where the i-th smallest of the
        // solver's values was.
        std::vector<HC> Cm(kk);
        for (int i = 0; i < k; ++i) {
            const int dst = perm[i];
            for (int r = 0; r < k; ++r) {
                HC acc = 0.0;
                for (int q = 0; q < k; ++q) acc += B[r + q * k] * Z[q + i * k];
                Cm[r + (size_t)dst * k] = acc;
                hv[(size_t)dst * 2 * k + r] = -acc;             // AW part
                hv[(size_t)dst * 2 * k + k + r] = th[i] * acc;  // W part
            }
            eval_[dst] = th[i];
        }
        // X = W Cm.  Real: one recombination launch into X.  Complex: per
        // column, ay = 0 - W (-Cm_c) with the update kernel, then a copy.
        if constexpr (kComplex) {
            std::vector<HC> neg(kk);
            for (size_t q = 0; q < kk; ++q) neg[q] = -Cm[q];
            CK(cudaMemcpyAsync(dG, neg.data(), sizeof(C) * kk, cudaMemcpyHostToDevice, st_));
            for (int cc = 0; cc < k; ++cc) {
                launch_update<C>(tabW, k, n_pad_, zero, Recur<C>{}, dG + (size_t)cc * k, ay, dout2, scratch_, st_);
                CK(cudaMemcpyAsync(X + (size_t)cc * ldx, ay, sizeof(C) * nrow_, cudaMemcpyDeviceToDevice, st_));
            }
            count_launch(k);
        } else {
            CK(cudaMemcpyAsync(dG, Cm.data(), sizeof(C) * kk, cudaMemcpyHostToDevice, st_));
            launch_ritz_out<double>(tabW, k, n_pad_, reinterpret_cast<const double *>(dG), k, k, X, ldx, nrow_,
                                    st_);
            count_launch();
        }
        CK(cudaMemcpyAsync(dh, hv.data(), sizeof(C) * 2 * kk, cudaMemcpyHostToDevice, st_));
        // r_c = 0 - [AW W] h_c = AW C_c - theta_c W C_c, |r_c|^2 -> dr2[c].
        for (int cc = 0; cc < k; ++cc)
            launch_update<C>(tabAWW, 2 * k, n_pad_, zero, Recur<C>{}, dh + (size_t)cc * 2 * k, ay, dr2 + cc, scratch_,
                             st_);
        count_launch(k);
        if (int e = gsum(dr2, (size_t)k)) return e;
        CK(cudaMemcpyAsync(r2.data(), dr2, sizeof(double) * k, cudaMemcpyDeviceToHost, st_));
        CK(cudaStreamSynchronize(st_));
        ++syncs_;
        worst = 0.0;
        for (int i = 0; i < k; ++i) {
            beta_[i] = std::sqrt(std::max(r2[i], 0.0));
            worst = std::max(worst, beta_[i]);
        }
        refined = true;
        if (worst <= tol_abs || pass + 1 == kRefinePasses) break;
        CK(cudaMemcpy2DAsync(Wb, vec * sizeof(C), X, ldx * sizeof(C), nrow_ * sizeof(C), k, cudaMemcpyDeviceToDevice,
                             st_));
    }
    if (!refined) return 0;
    if (!user_dev_) {
        const size_t ue = sizeof(User);
        CK(host_copy_2d(evec_, ue * lde_, X, ue * n_pad_, ue * nrow_, k, cudaMemcpyDeviceToHost, st_));
    }
    *max_res = worst;
    return 0;
}

template <class T>
void Engine<T>::log_progress() {
    if (info_->verbose <= 0) return;
    LogOut log(info_);
    FILE *fp = log.fp;
    std::fprintf(fp, "MATVEC: %10d,    Nloop: %10d,     Nec: %10d\n", info_->matvec, info_->nloop, info_->nec);
    std::fprintf(fp, "Reorth: %10d,    Nrand: %10d,    Ierr: %10d\n", info_->north, info_->nrand, info_->stat);
    std::fprintf(fp, "Target: %10.3e,   ResNrm: %10.3e,  CFact: %10.3e\n", info_->trgt, info_->tres, info_->crat);
}

template <class T>
void Engine<T>::run() {
    trl_info *info = info_;
    const double t_start = now_s();
    int locked = info->nec;
    if (locked > 0) {
        for (int i = 0; i < locked; ++i) {
            alpha_[i] = eval_[i];
            beta_[i] = 0.0;
        }
    }
    int jnd = 0;
    int stat = initial_guess(&jnd);
    int kept = jnd;
    info->stat = stat;
    if (stat != 0) {
        final_j1_ = 0;
        return;
    }
    int i1 = info->ned - jnd;
    int next_test = i1 + std::min(i1, std::min(6, info->ned / 2));
    int chkpnt = info->cpflag <= 0 ? info->maxmv + info->maxlan : info->maxmv / info->cpflag;
    int prek = kept;
    int j1 = kept;  // columns that map to the caller's evec on exit

    while (info->matvec < info->maxmv && info->nec < info->ned) {
        // ---- steps from the (re)start on, the arrowhead one first -------------
        int acc = 0;
        long run = 0;
        if (spec_enabled()) {
            // Up to the next convergence test, which never comes right after
            // the first step.
            run = std::min<long>((long)info->klan - jnd, std::max<long>(2, (long)next_test - info->matvec));
            const bool sweep = sweeps(jnd);
            if (sweep) run = std::min<long>(run, kSweepCols + 1 - jnd);
            run = std::min<long>(run, streak_ / 2);
            if (run >= 2 && (sweep || coop_steps(jnd, (int)run))) acc = spec_segment(&jnd, (int)run, kept);
            if (acc < 0) {
                stat = acc;
                break;
            }
        }
        if (acc == 0) {
            // ---- first step after (re)start: arrowhead coupling -------------------
            jnd++;
            if (jnd + 1 > maxlan_ + 1 || jnd + 1 >= P_) {
                stat = -1111;
                break;
            }
            // FP64 views of the current vector and the output slot.
            if constexpr (kWide) {
                qa64_ = reinterpret_cast<C *>(col(jnd - 1));
                qb64_ = jnd >= 2 ? reinterpret_cast<C *>(col(jnd - 2)) : nullptr;
                r64_ = reinterpret_cast<C *>(col(jnd));
            }
            tm_begin();
            if ((stat = apply_op(qa64_, r64_, true))) break;
            tm_mid();
            // Coefficients (beta_0 .. beta_{jnd-2}, alpha_{jnd-1}); the device
            // writes alpha into the last slot before the coupling update.
            {
                std::vector<C> g(jnd);
                for (int i = 0; i < jnd - 1; ++i) {
                    if constexpr (kComplex)
                        g[i] = zd{beta_[i], 0.0};
                    else
                        g[i] = beta_[i];
                }
                if constexpr (kComplex)
                    g[jnd - 1] = zd{0.0, 0.0};
                else
                    g[jnd - 1] = 0.0;
                if (cudaMemcpyAsync(d_coef_, g.data(), sizeof(C) * jnd, cudaMemcpyHostToDevice, st_) != cudaSuccess) {
                    stat = -1001;
                    break;
                }
                cudaMemcpyAsync(reinterpret_cast<double *>(d_coef_ + (jnd - 1)), d_scal_ + kAlpha, sizeof(double),
                                cudaMemcpyDeviceToDevice, st_);
                Recur<C> none;
                int pid = pbeg();
                launch_update<T>(d_cols_, jnd, n_pad_, r64_, none, d_coef_, r64_, d_scal_ + kR2Post, scratch_, st_);
                pend(pid, TRLX_K_UPDATE, (double)jnd * nrow_ * sv() + 2.0 * nrow_ * cs());
                count_launch();
                cudaStreamSynchronize(st_);  // g must outlive the copy
            }
            fl_ += 2 * jnd * nrow_ + nrow_ + nrow_;
            double f0 = fl_;
            const int passes = info->north;
            stat = orth(jnd, false, 0.0, kept);
            took_steps(1, info->north == passes + 1);
            fl_h_ += fl_ - f0;
            tm_end();
            if (stat) break;
            rotate_fp64();
        }
        // Arrow -> tridiagonal for the non-locked part (the columns up to and
        // with the first step's).
        for (int i = 0; i < locked; ++i) {
            alfrot_[i] = alpha_[i];
            betrot_[i] = 0.0;
        }
        i1 = kept + 1 - locked;
        arrow_to_tridiag(i1, &alpha_[locked], &beta_[locked], rot_.data(), &alfrot_[locked], &betrot_[locked]);
        fl_ += 8 * i1 * i1 * i1 / 3;
        betrot_[kept] = beta_[kept];

        // ---- regular Lanczos steps ---------------------------------------------
        auto test_convergence = [&]() -> int {
            int st2 = get_eval(jnd, locked, alfrot_.data(), betrot_.data(), lambda_.data(), res_.data());
            if (st2) return st2;
            track_ritz(jnd);
            const int ne = std::min(mev_, jnd);
            std::memcpy(eval_, lambda_.data(), sizeof(double) * ne);
            convergence_test(jnd, lambda_.data(), res_.data(), info, wrk2_.data());
            if (info->nec < info->ned && info->nec > 0) {
                next_test = (int)((double)(info->ned * info->matvec) / (double)info->nec);
            } else if (info->nec == 0) {
                next_test = next_test + next_test;
                if (info->maxlan == info->ntot) next_test = (int)std::ceil(0.5 * (info->maxlan + info->matvec));
            }
            log_progress();
            return 0;
        };
        if (acc > 1 && acc == run && info->matvec >= next_test && (stat = test_convergence())) break;
        while (jnd < info->klan && info->nec < info->ned) {
            if (spec_enabled()) {
                // Steps up to the next convergence test (or the restart).
                long S = (long)info->klan - jnd;
                const bool sweep = sweeps(jnd);
                if (sweep) S = std::min<long>(S, kSweepCols + 1 - jnd);
                if (next_test > info->matvec) S = std::min<long>(S, (long)next_test - info->matvec);
                else S = 1;
                S = std::min<long>(S, streak_ / 2);
                // A single step pays as a cooperative run only, the discrete
                // kernels need a column before the last.
                if (S >= 2 ? sweep || (kWide && jnd >= 2) || coop_steps(jnd, (int)S)
                           : S == 1 && coop_steps(jnd, (int)S)) {
                    const int acc = spec_segment(&jnd, (int)S, kept);
                    if (acc < 0) {
                        stat = acc;
                        break;
                    }
                    if (acc == S) {
                        if (info->matvec >= next_test && (stat = test_convergence())) break;
                        continue;
                    }
                    if (jnd >= info->klan) break;
                }
            }
            jnd++;
            if (jnd + 1 >= P_) {
                stat = -1111;
                break;
            }
            if constexpr (kWide) {
                qa64_ = reinterpret_cast<C *>(col(jnd - 1));
                qb64_ = reinterpret_cast<C *>(col(jnd - 2));
                r64_ = reinterpret_cast<C *>(col(jnd));
            }
            tm_begin();
            if ((stat = apply_op(qa64_, r64_, true))) break;
            tm_mid();
            fl_ += 6 * nrow_;
            double f1 = fl_;
            const int passes = info->north;
            stat = orth(jnd, true, beta_[jnd - 2], kept);
            took_steps(1, info->north == passes + 1);
            fl_h_ += fl_ - f1;
            tm_end();
            alfrot_[jnd - 1] = alpha_[jnd - 1];
            betrot_[jnd - 1] = beta_[jnd - 1];
            if (stat) break;
            rotate_fp64();
            if (info->matvec >= next_test && (stat = test_convergence())) break;
        }
        if (stat) break;

        // ---- restart or finish -------------------------------------------------
        const double t_r0 = now_s();
        const double fr0 = fl_;
        prek = kept;
        const int jml = jnd - locked;
        int i2 = kept - locked + 1;
        const bool solved = info->nec < info->ned;
        if (solved) {
            if ((stat = tridiag_.get_eval(jnd, locked, alfrot_.data(), betrot_.data(), lambda_.data(), res_.data())))
                break;
            track_ritz(jnd);
            convergence_test(jnd, lambda_.data(), res_.data(), info, wrk2_.data());
            log_progress();
        }
        if (info->nec < info->ned && info->matvec < info->maxmv) {
            shuffle_eig(jml, info->klan - locked, &lambda_[locked], &res_[locked], info, &kept, locked);
            tridiag_.vectors(i2, rot_.data(), kept, &lambda_[locked], yy_.data());
            if (locked + kept > 0) std::memcpy(alpha_.data(), lambda_.data(), sizeof(double) * (locked + kept));
            for (int i = 0; i < kept; ++i) beta_[locked + i] = yy_[(size_t)(i + 1) * jml - 1] * betrot_[jnd - 1];
            if (jml > info->ned + (info->ned / 5 + 6))
                set_locking(jml, kept, &alpha_[locked], &beta_[locked], yy_.data(), info->anrm, &i2);
            else
                i2 = 0;
            if ((stat = restart_ritz(locked, jml, kept, jnd))) break;
            fl_ += 2 * nrow_ * jml * kept;
            kept += locked;
            locked += i2;
            info->locked = locked;
            jnd = kept;
            if (jnd > mev_ && jnd - mev_ >= std::max(1, info->maxlan - mev_ + 1) - 1) {
                stat = -1111;
                break;
            }
            if (info->nec > 0)
                next_test = (int)(((double)(info->matvec * info->ned)) / ((double)info->nec));
            else
                next_test = next_test + info->maxlan;
            const int ne = std::min(mev_, jnd);
            if (ne > 0) std::memcpy(eval_, lambda_.data(), sizeof(double) * ne);
            j1 = std::min(jnd, mev_);
            if (info->matvec >= chkpnt) {
                // Kept vectors 0..jnd-1 and the residual (column jnd; its
                // FP64 copy is q_cur for a 32-bit basis).
                const int kj = jnd;
                stat = write_checkpoint(kj, [&](int i) -> const C * {
                    if constexpr (kWide) {
                        return reinterpret_cast<const C *>(col(i));
                    } else {
                        if (i == kj) return qa64_;
                        launch_load<T>(col(i), n_pad_, r64_, st_);
                        return r64_;
                    }
                });
                if (stat) break;
                chkpnt += info->maxmv / std::max(info->cpflag, 1);
            }
        } else {
            kept = std::min(info->nec, std::max(info->ned, mev_ - 1));
            info->nec = kept;
            if (kept == 0) kept = std::min(mev_ - 1, info->ned);
            sort_eig(jnd, info->lohi, kept, info->ref, lambda_.data(), res_.data());
            std::memcpy(eval_, lambda_.data(), sizeof(double) * kept);
            int tstat = 0;
            if (solved && locked == 0)
                tridiag_.vectors(i2, rot_.data(), kept, eval_, yy_.data());
            else if (kept * 3 < jnd)
                tstat = get_tvec(jnd, alfrot_.data(), betrot_.data(), locked, i2, rot_.data(), kept, eval_, yy_.data());
            if ((!(solved && locked == 0) && kept * 3 >= jnd) || tstat != 0) {
                tstat = get_tvec_a(jnd, prek, alpha_.data(), beta_.data(), kept, eval_, yy_.data());
                if (tstat) {
                    stat = tstat;
                    break;
                }
            }
            if (kept > 0) std::memcpy(alpha_.data(), eval_, sizeof(double) * kept);
            for (int i = 0; i < kept; ++i) beta_[i] = betrot_[jnd - 1] * yy_[(size_t)(1 + i) * jnd - 1];
            if ((stat = final_vectors(jnd, kept))) break;
            fl_ += 2 * nrow_ * jml * kept;
            jnd = kept;
            j1 = kept;
        }
        t_res_ += now_s() - t_r0;
        fl_r_ += fl_ - fr0;
        info->nloop++;
    }
    final_j1_ = j1;
    info->stat = stat;
    tm_collect(true);
    double max_res = -1.0;
    const bool want_refine = opt_.refine > 0 || (opt_.refine < 0 && !kWide);
    if (want_refine && stat == 0 && info->nec > 0 && info->lohi != 0) {
        const double tr0 = now_s();
        const int rs = refine_fp64(std::min(info->nec, j1), &max_res);
        t_res_ += now_s() - tr0;
        if (rs) info->stat = rs;
    }
    // Flop counts go to the floating-point counters (the int ones would
    // overflow at these sizes); timers are seconds in the tick_* fields.
    info->rflp += fl_;
    info->rflp_h += fl_h_;
    info->rflp_r += fl_r_;
    info->tick_o += t_op_;
    info->tick_h += t_orth_;
    info->tick_r += t_res_;
    auto &s = last_stats();
    s.seconds_total = now_s() - t_start;
    s.seconds_op = t_op_;
    s.seconds_orth = t_orth_;
    s.seconds_restart = t_res_;
    s.kernel_launches = launches_;
    s.cgs_passes = info->north;
    s.host_syncs = syncs_;
    s.max_true_residual = max_res;
    s.op_bytes = builtin_ ? spmv_bytes(builtin_) * info->matvec : 0.0;
    cudaStreamSynchronize(st_);
    flush_prof();
    for (int k = 0; k < 8; ++k) {
        s.kernel_seconds[k] = kt_[k];
        s.kernel_bytes[k] = kb_[k];
        s.kernel_count[k] = kc_[k];
    }
    s.basis_bytes = kb_[TRLX_K_PROJECT] + kb_[TRLX_K_UPDATE] + kb_[TRLX_K_RITZ];
    s.seconds_setup = setup_seconds_;
    s.speculative_steps = spec_accepted_;
    s.speculative_discarded = discarded_;
}

template <class T>
void solve(typename Engine<T>::OpFn op, trl_uo uo, trl_info *info, int nrow, int mev, double *eval,
           typename Engine<T>::User *evec, int lde, double *res_out, int res_len, const Options &opt) {
    Engine<T> eng(op, uo, info, nrow, mev, eval, evec, lde, opt);
    int st = eng.setup();
    if (st) {
        info->stat = st;
        return;
    }
    eng.run();
    if (res_out) eng.residual_output(res_out, res_len);
}

}  // namespace

void clear_counter(trl_info *info, int nrow, int mev, int lde) {
    info->stat = 0;
    if (nrow != info->nloc || nrow > info->ntot) {
        std::printf("TRLAN: info not setup for this problem.\n");
        std::printf("       Please reset info before calling TRLAN.\n");
        info->stat = -1;
    }
    if (info->nec < 0) info->nec = 0;
    if (lde < nrow) {
        std::printf("TRLAN: leading dimension of EVEC to small.\n");
        info->stat = -2;
    }
    if (info->tol >= 1.0)
        info->tol = std::sqrt(DBL_EPSILON);
    else if (info->tol <= DBL_MIN)
        info->tol = DBL_EPSILON;
    if (info->ned + info->ned >= info->ntot) {
        std::printf("TRLAN: info->ned (%d) is large relative to the matrix dimension (%d)\n", info->ned,
                    info->ntot);
        std::printf(" **    It is more appropriate to use LAPACK dsyev/ssyev.\n");
        if (info->ned > info->ntot) {
            info->ned = std::min(info->ntot - 1, info->maxlan - 3);
            std::printf("TRLAN: ** reduced ned to %d **\n", info->ned);
        }
    }
    if (mev < info->ned) {
        std::printf("TRLAN: array EVAL and EVEC can not hold wanted number of eigenpairs.\n");
        info->stat = -3;
    }
    if (info->ntot < 10) {
        std::printf("TRLAN is not designed to work with such a small matrix(%dx%d).  Please use LAPACK or "
                    "EISPACK instead.\n",
                    info->ntot, info->ntot);
        info->stat = -4;
    }
    if (info->maxlan < info->ned + 3) {
        info->maxlan = info->ned + std::min(info->ned, 20) + (int)std::log((double)info->ntot);
        info->maxlan = std::min(info->maxlan, info->ntot);
        std::printf("TRLAN: ** reset maxlan to %d! **\n", info->maxlan);
    }
    if (info->maxlan < mev) {
        int ntmp = std::min(info->ntot, std::max(100 + info->ned, 10 * info->ned));
        info->maxlan = mev < ntmp ? mev : ntmp;
    }
    if (info->maxlan < 5) {
        std::printf("TRLAN must have at least 5 basis vectors, it is currently %d.\n", info->maxlan);
        info->stat = -5;
    }
    info->tmv = -1;
    info->klan = std::min(info->maxlan, info->ntot);
    if (info->restart >= 7) info->klan = std::min(info->maxlan, std::max(100, std::min(info->klan, 2 * info->ned)));
    info->locked = info->nec;
    info->matvec = 0;
    info->nloop = 0;
    info->north = 0;
    info->nrand = 0;
    info->flop = 0;
    info->rflp = 0;
    info->flop_h = 0;
    info->rflp_h = 0;
    info->flop_r = 0;
    info->rflp_r = 0;
    info->tick_t = 0.0;
    info->clk_op = 0;
    info->tick_o = 0.0;
    info->clk_orth = 0;
    info->tick_h = 0.0;
    info->clk_res = 0;
    info->tick_r = 0.0;
    info->clk_in = 0;
    info->clk_out = 0;
    info->wrds_in = 0;
    info->wrds_out = 0;
    info->avgm = 0.0;
}

void run_trlan(trl_matvec op, trl_uo uo, trl_info *info, int nrow, int mev, double *eval, double *evec, int lde,
               int lwrk, double *wrk, const Options &opt) {
    const double t0 = now_s();
    last_stats() = trlx_stats{};
    if (info->ned > mev) {
        std::printf("info->ned (%d) is larger than mev (%d) reducing info->ned to %d\n", info->ned, mev, mev);
        info->ned = mev;
    }
    if (info->ned <= info->nec || info->ned <= 0) return;
    info->stat = 0;
    clear_counter(info, nrow, mev, lde);
    if (info->stat != 0) return;
    { LogOut start(info, "w"); }  // a new solve starts a new log file (SRC/trlan.c:235)
    if (opt.basis_bits == 32)
        solve<float>(op, uo, info, nrow, mev, eval, evec, lde, wrk, std::min(mev, lwrk), opt);
    else
        solve<double>(op, uo, info, nrow, mev, eval, evec, lde, wrk, std::min(mev, lwrk), opt);
    info->tick_t += now_s() - t0;
}

void run_ztrlan(ztrl_matvec op, trl_info *info, int nrow, int mev, double *eval, trl_dcomplex *evec, int lde,
                trl_dcomplex *misc, int nmis, const Options &opt) {
    const double t0 = now_s();
    last_stats() = trlx_stats{};
    if (info->ned > mev) {
        std::printf("info->ned (%d) is larger than mev (%d) reducing info->ned to %d\n", info->ned, mev, mev);
        info->ned = mev;
    }
    if (info->ned <= info->nec || info->ned <= 0) return;
    info->stat = 0;
    clear_counter(info, nrow, mev, lde);
    if (info->stat != 0) return;
    { LogOut start(info, "w"); }  // a new solve starts a new log file (SRC/trlan.c:235)
    std::vector<double> res(mev, 0.0);
    if (opt.basis_bits == 32)
        solve<zf>(op, nullptr, info, nrow, mev, eval, evec, lde, res.data(), mev, opt);
    else
        solve<zd>(op, nullptr, info, nrow, mev, eval, evec, lde, res.data(), mev, opt);
    if (misc && nmis > 0) {
        for (int i = 0; i < std::min(mev, nmis); ++i) misc[i] = trl_dcomplex{res[i], 0.0};
    }
    info->tick_t += now_s() - t0;
}

}  // namespace trlb
