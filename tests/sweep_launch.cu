// One launch_sweep (kernels/sweep.cu), for a test against fake_cudart.cpp.
#include "kernels/sweep.h"

extern "C" int sweep_status() {
    trlb::Scratch s;
    s.max_blocks = 148;
    static double partials[148 * 8];
    static unsigned tickets[64];
    s.partials = partials;
    s.tickets = tickets;
    trlb::SweepArgs<double> a;
    a.k = 4;
    a.n_pad = 1 << 17;
    return trlb::launch_sweep<double>(a, s, nullptr);
}
