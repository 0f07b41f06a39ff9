// paired_work.cu -- the item list a paired stage kernel would walk, from its
// argument, and an item as the kernel reads it; the one part of the host
// runtime (fake_cuda.cpp) that needs the kernels' header.
#include "../../copara-cgfd3d_b200/csrc/stage_pair_impl.cuh"

extern "C" const int4 *paired_items(const void *work, int list, int *n) {
  const cgfd::pair::Work &wk = *static_cast<const cgfd::pair::Work *>(work);
  const bool lean = list == cgfd::pair::LEAN_BOTH;
  *n = wk.nitems[lean];
  return wk.items[lean];
}
extern "C" void paired_item(const int4 *packed, int *v) {
  const cgfd::pair::Item t = cgfd::pair::unpack_item(*packed);
  v[0] = t.i0, v[1] = t.j0, v[2] = t.z0, v[3] = t.z1, v[4] = t.model, v[5] = t.part;
}
