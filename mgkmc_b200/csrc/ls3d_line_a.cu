// Instantiations of the 3D iteration kernels (ls3d_line.cuh), lengths 24 27 32 36 48 54.
#include "ls3d_line.cuh"

namespace mgk {
const Ls3Line* ls3_line_a(int n, int prec) {
  switch (n) {
    case 24: return prec == MGK_FP64 ? ls3_make<double, 24, true>() : nullptr;
    case 27: return prec == MGK_FP64 ? ls3_make<double, 27, true>() : nullptr;
    case 32: return prec == MGK_FP64 ? ls3_make<double, 32, true>() : nullptr;
    case 36: return prec == MGK_FP64 ? ls3_make<double, 36, true>() : nullptr;
    case 48: return prec == MGK_FP64 ? ls3_make<double, 48, true>() : nullptr;
    case 54: return prec == MGK_FP64 ? ls3_make<double, 54, true>() : nullptr;
    default: return nullptr;
  }
}
}  // namespace mgk
