// Cooperative kernel for runs of Lanczos steps on short vectors (coop.cu).
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

struct trlx_operator;

namespace trlb {

template <class C>
struct CoopArgs {
    int nrow;
    long n_pad;
    int chunk;       // rows per block (multiple of 32)
    int kmax;        // columns the shared arrays hold
    int nres;        // basis columns kept in shared memory
    int ecap;        // operator entries kept in shared memory per block (0: none)
    const long long *ptr;  // CSR row pointers, or SELL-C-32 slice pointers
    int sell;
    int tpr;         // lanes per row of the product (a power of two)
    int wide;        // rows of more entries get a warp
    const int *ci;
    const C *va;
    C *const *cols;  // basis column table
    C *z[2];         // exchange vectors (n_pad rows each)
    int j0, S;       // steps j0 + 1 .. j0 + S
    int kept;        // leading columns coupled only to column `kept`
    const double *ta, *tb;  // alphas and betas of the first j0 columns
    double *log;     // [s][4]: alpha, |r|^2 before, |h|^2, |r|^2 after (s = 1..S)
    double *failed;  // set to 1 when a barrier gave up
    double *part;    // two sets of the clusters' partial sums
    unsigned *sync;  // two counters, zero between launches
    long polls;      // of the grid barrier before it gives up
};

constexpr long kCoopPolls = 1L << 22;  // some seconds

// Whether the kernel takes runs of this operator, up to `kmax` columns, on the
// current device: CSR or unsorted SELL, sizes that fit in shared memory,
// cooperative launches.
template <class C>
bool coop_applies(const trlx_operator *A, long n_pad, int kmax, size_t part_doubles);

// Runs S steps of a built-in CSR operator or an unsorted SELL one.  Returns
// 0, or -1 if the kernel does not apply (operator form, device, sizes) or was
// not launched (nothing is changed then).
template <class C>
int launch_coop(const trlx_operator *A, C *const *cols, C *z0, C *z1, long n_pad, int j0, int S, int kept,
                const double *ta, const double *tb, double *log, double *failed, double *part, size_t part_doubles,
                unsigned *sync, long polls, cudaStream_t st);

}  // namespace trlb
