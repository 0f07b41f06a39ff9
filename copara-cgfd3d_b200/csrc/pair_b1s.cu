// pair_b1s.cu -- the paired stage kernels over the stress part of the general items,
// RK stage kind 1 (inner stages), BF16 storage, for the 8 stencil directions,
// single-model and batched.
#include "stage_pair_impl.cuh"

cgfd::pair::Entry cgfd::pair::entry_b1s() { return make_entry<__nv_bfloat16, 1, GEN_STR>(); }
