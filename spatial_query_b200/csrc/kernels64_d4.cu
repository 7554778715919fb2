// Kernel instantiations of f64 scenes for D = 4.
#include "traverse.cuh"

namespace sq {
bool kernel_set64_d4(int narrow, KernelSet* out) {
  switch (narrow) {
    case kNarrowAabb: *out = make_kernel_set64<4, kNarrowAabb>(); return true;
    case kNarrowSphere: *out = make_kernel_set64<4, kNarrowSphere>(); return true;
    case kNarrowSphereNear: *out = make_kernel_set64<4, kNarrowSphereNear>(); return true;
    default: return false;
  }
}
}  // namespace sq
