// Instantiations of the 3D iteration kernels (ls3d_line.cuh), lengths 108 128 144 162.
#include "ls3d_line.cuh"

namespace mgk {
const Ls3Line* ls3_line_c(int n, int prec) {
  switch (n) {
    case 108: return prec == MGK_FP64 ? ls3_make<double, 108, true>() : nullptr;
    case 128: return prec == MGK_FP64 ? ls3_make<double, 128, true>() : ls3_make<float, 128, false>();
    case 144: return prec == MGK_FP64 ? ls3_make<double, 144, true>() : nullptr;
    case 162: return prec == MGK_FP64 ? ls3_make<double, 162, true>() : nullptr;
    default: return nullptr;
  }
}
}  // namespace mgk
