// pair_h0v.cu -- the paired stage kernels over the velocity part of the general items,
// RK stage kind 0 (first stage), FP16 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_h0v() { return make_entry<__half, 0, GEN_VEL>(); }
