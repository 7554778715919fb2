// Kernel instantiations of f64 scenes for D = 3.
#include "traverse.cuh"

namespace sq {
bool kernel_set64_d3(int narrow, KernelSet* out) {
  switch (narrow) {
    case kNarrowAabb: *out = make_kernel_set64<3, kNarrowAabb>(); return true;
    case kNarrowSphere: *out = make_kernel_set64<3, kNarrowSphere>(); return true;
    case kNarrowSphereNear: *out = make_kernel_set64<3, kNarrowSphereNear>(); return true;
    case kNarrowTri: *out = make_kernel_set64<3, kNarrowTri>(); return true;
    default: return false;
  }
}
}  // namespace sq
