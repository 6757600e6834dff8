// TridiagVectors (host/dense.h) for a test.
#include "dense.h"

extern "C" int tridiag_vectors(int nd, int locked, const double *alpha, const double *beta, int nrot,
                               const double *rot, int nlam, double *lambda, double *res, double *yy) {
    trlb::TridiagVectors t;
    const int e = t.get_eval(nd, locked, alpha, beta, lambda, res);
    if (e == 0) t.vectors(nrot, rot, nlam, lambda + locked, yy);
    return e;
}
