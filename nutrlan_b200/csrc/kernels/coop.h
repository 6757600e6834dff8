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
    int lanes;       // log2 of the lanes per row of the product
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

// Operators of at least so many rows take their steps as sweeps (sweep.h):
// the basis leaves L2, and the cooperative kernel reads it twice a step.
// Lattice, 5 entries a row, cooperative / sweeps, a call: 123904 rows, 48
// columns 3.3 / 3.7 ms, 96 columns 5.4 / 6.0; 186624 rows 4.3 / 4.2, 9.2 / 7.0.
// (Complex: 65536 rows 3.4 / 4.5 and 6.3 / 7.2, 92416 rows 4.8 / 4.5 and 11.7 / 7.6;
// four launches a step 7.6 and 13.1.)
constexpr long kCoopRows = 1L << 17;
// So do operators of more doubles than this to gather in a product: the
// cooperative kernel gathers from two vectors.  Random columns, 48 columns,
// cooperative / sweeps / four launches a step, a call: 98304 rows of 17
// entries 6.3 / 4.9 / 6.8 ms, of 33 9.4 / 6.0 / 8.5, of 65 20.1 / 11.3 / 13.7;
// 32768 rows of 33 3.3 / 3.7 / 5.5, of 129 7.1 / 5.0 / 6.8.  (Band matrices
// lose some there: 98304 rows of 33, 64 columns, 5.4 / 6.5 / 9.0.)
constexpr long long kCoopWords = 1500000;

// Whether a run of this operator is better off in the cooperative kernel than
// in sweeps, by rows and entries.  The product kernels that sweeps alternate
// with leave a row to one lane (SELL) or eight (CSR), so that a long row
// outweighs the second gather: 98304 rows of 33 entries, one of 3000 12.5 /
// 10.2 ms, of 10000 15.6 / 18.2; SELL, 17 entries, longest 300 8.5 / 16.3.
template <class C>
bool coop_pays(const trlx_operator *A, long n_pad);

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
