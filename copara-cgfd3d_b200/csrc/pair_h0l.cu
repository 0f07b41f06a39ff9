// pair_h0l.cu -- the paired stage kernels over the lean items,
// RK stage kind 0 (first stage), FP16 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_h0l() { return make_entry<__half, 0, LEAN_BOTH>(); }
