// paired_work.cu -- the item list a paired stage kernel would walk, from its
// argument; the one part of the host runtime (fake_cuda.cpp) that needs the
// kernels' header.
#include "../../copara-cgfd3d_b200/csrc/stage_pair_impl.cuh"

extern "C" const int4 *paired_items(const void *work, int list, int *n) {
  const cgfd::pair::Work &wk = *static_cast<const cgfd::pair::Work *>(work);
  const bool lean = list == cgfd::pair::LEAN_BOTH;
  *n = wk.nitems[lean];
  return wk.items[lean];
}
