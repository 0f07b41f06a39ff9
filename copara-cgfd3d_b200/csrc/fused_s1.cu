// fused_s1.cu -- instantiates the stress kernels of RK stage kind 1
// (inner stages) for the 8 stencil directions.
#include "stage_fused_impl.cuh"

namespace cgfd {
namespace fused {

void launch_s1(const Plan &pl, const StageMaps &m, const StageArgs &a, int *err,
                  cudaStream_t s) {
  launch_dirs<PART_STR, 1>(pl, m, a, err, s);
}

cudaError_t attrs_s1() { return set_attrs<PART_STR, 1>(); }

int resident_str() { return resident_ctas<PART_STR>(); }

}  // namespace fused
}  // namespace cgfd
