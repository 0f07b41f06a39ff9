// pair_f2s.cu -- the paired stage kernels over the stress part of the general items,
// RK stage kind 2 (final stage), FP32 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_f2s() { return make_entry<float, 2, GEN_STR>(); }
