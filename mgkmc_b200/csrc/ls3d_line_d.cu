// Instantiations of the 3D iteration kernels (ls3d_line.cuh), lengths 192 216 243 256.
#include "ls3d_line.cuh"

namespace mgk {
const Ls3Line* ls3_line_d(int n, int prec) {
  switch (n) {
    case 192: return prec == MGK_FP64 ? ls3_make<double, 192, true>() : nullptr;
    case 216: return prec == MGK_FP64 ? ls3_make<double, 216, true>() : nullptr;
    case 243: return prec == MGK_FP64 ? ls3_make<double, 243, true>() : nullptr;
    case 256: return prec == MGK_FP64 ? ls3_make<double, 256, true>() : nullptr;
    default: return nullptr;
  }
}
}  // namespace mgk
