// pair_f2v.cu -- the paired stage kernels over the velocity part of the general items,
// RK stage kind 2 (final stage), FP32 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_f2v() { return make_entry<float, 2, GEN_VEL>(); }
