// Kernel instantiations of f64 scenes for D = 2.
#include "traverse.cuh"

namespace sq {
bool kernel_set64_d2(int narrow, KernelSet* out) {
  switch (narrow) {
    case kNarrowAabb: *out = make_kernel_set64<2, kNarrowAabb>(); return true;
    case kNarrowSphere: *out = make_kernel_set64<2, kNarrowSphere>(); return true;
    case kNarrowSphereNear: *out = make_kernel_set64<2, kNarrowSphereNear>(); return true;
    default: return false;
  }
}
}  // namespace sq
