// rk4_pair.cuh -- the paired-pass transient kernel's launcher (rk4_pair.cu),
// called by rk4_krylov.cu.
#pragma once
#include "fast_common.cuh"

namespace hsb {

// resources for the model if the kernel takes it (*taken: w->kfn is set)
int pair_prepare(hsb_dev_model *m, FastWork *w, bool *taken);
bool pair_is_kernel(const void *fn);
// the launch and the copy of its counters to the host, without waiting
int pair_enqueue(hsb_dev_model *m, FastWork *w, double T, hsb_stats *st, const double *bpow, int K);

}  // namespace hsb
