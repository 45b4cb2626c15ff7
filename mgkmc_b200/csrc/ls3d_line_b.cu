// Instantiations of the 3D iteration kernels (ls3d_line.cuh), lengths 64 72 81 96.
#include "ls3d_line.cuh"

namespace mgk {
const Ls3Line* ls3_line_b(int n, int prec) {
  switch (n) {
    case 64: return prec == MGK_FP64 ? ls3_make<double, 64, true>() : ls3_make<float, 64, false>();
    case 72: return prec == MGK_FP64 ? ls3_make<double, 72, true>() : nullptr;
    case 81: return prec == MGK_FP64 ? ls3_make<double, 81, true>() : nullptr;
    case 96: return prec == MGK_FP64 ? ls3_make<double, 96, true>() : ls3_make<float, 96, false>();
    default: return nullptr;
  }
}
}  // namespace mgk
