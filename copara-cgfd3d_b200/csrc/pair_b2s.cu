// pair_b2s.cu -- the paired stage kernels over the stress part of the general items,
// RK stage kind 2 (final stage), BF16 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_b2s() { return make_entry<__nv_bfloat16, 2, GEN_STR>(); }
