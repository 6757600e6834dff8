// One launch_coop (kernels/coop.cu) on `rows` rows, for a test against fake_cudart.cpp.
#include "kernels/coop.h"
#include "kernels/spmv.h"

extern "C" int coop_status(int rows) {
    trlx_operator A;
    A.kind = 0;
    A.nrow = rows;
    A.nnz = rows;
    return trlb::launch_coop<double>(&A, nullptr, nullptr, nullptr, rows, 2, 4, 0, nullptr, nullptr, nullptr, nullptr,
                                     nullptr, 1 << 20, nullptr, trlb::kCoopPolls, nullptr);
}
