// Single-sweep Lanczos steps (sweep.cu): the Gram-Schmidt update of one
// vector and the projection of the next in one pass over the basis.
#pragma once

#include <cuda_runtime.h>

#include "lanczos_kernels.h"

namespace trlb {

// Columns a sweep takes (8 warps of 16).
constexpr int kSweepCols = 128;

// Device state of a run of sweeps; column indices are those of the basis.
template <class T>
struct SweepArgs {
    using C = typename Store<T>::C;
    T *const *cols = nullptr;  // column table
    const T *pool = nullptr;   // the allocation that holds the columns (at most 64 GB)
    int k = 0;                 // columns 0 .. k-1 are finished, this sweep makes column k
    int kept = 0;              // leading columns coupled only to column `kept` (arrowhead part of T)
    int first = 0;             // 1: x already is column k (nothing to correct or store)
    long n_pad = 0;
    C *x = nullptr;         // in: r, not yet orthogonalised (unnormalised); out: q_k (FP64)
    C *y = nullptr;         // in: A r; out: the next r
    const C *xp = nullptr;  // 32-bit storage: q_{k-1} in FP64; else null
    const double *dot = nullptr;  // Re(r^H A r)
    // Read by the sweep and rewritten for the next one by its last block:
    C *a = nullptr;         // h = V^H r (k values)
    C *c = nullptr;         // T h (+ beta^2 on its last entry for 64-bit storage)
    double *ta = nullptr, *tb = nullptr;  // alphas and betas of T so far
    double *sc = nullptr;   // 1 / beta, beta^2, beta of the recurrence for 32-bit storage
    double *lg = nullptr;   // log of step k + 1: alpha, |r|^2 before the pass, |h|^2, |r|^2 after
    double *lg_prev = nullptr;  // log of step k (its last entry is written here)
};

// 0, or -1 if the kernel was not launched (nothing is changed then).
template <class T>
int launch_sweep(const SweepArgs<T> &a, Scratch &s, cudaStream_t st);

}  // namespace trlb
