// Instantiations of the 2D iteration kernels (ls2d_line.cuh), lengths 288 324 384 432.
#include "ls2d_line.cuh"

namespace mgk {
const Ls2Line* ls2_line_e(int n, int kind) {
  switch (n) {
    case 288: return ls2_pick<288>(kind);
    case 324: return ls2_pick<324>(kind);
    case 384: return ls2_pick<384>(kind);
    case 432: return ls2_pick<432>(kind);
    default: return nullptr;
  }
}
}  // namespace mgk
