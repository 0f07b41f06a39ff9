// pair_f1l.cu -- the paired stage kernels over the lean items,
// RK stage kind 1 (inner stages), FP32 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_f1l() { return make_entry<float, 1, LEAN_BOTH>(); }
