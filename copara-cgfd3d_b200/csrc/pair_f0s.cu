// pair_f0s.cu -- the paired stage kernels over the stress part of the general items,
// RK stage kind 0 (first stage), FP32 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_f0s() { return make_entry<float, 0, GEN_STR>(); }
