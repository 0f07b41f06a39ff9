// pair_f0v.cu -- the paired stage kernels over the velocity part of the general items,
// RK stage kind 0 (first stage), FP32 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_f0v() { return make_entry<float, 0, GEN_VEL>(); }
