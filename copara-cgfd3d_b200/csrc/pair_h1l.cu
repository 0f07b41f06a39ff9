// pair_h1l.cu -- the paired stage kernels over the lean items,
// RK stage kind 1 (inner stages), FP16 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_h1l() { return make_entry<__half, 1, LEAN_BOTH>(); }
