// Instantiations of the 2D iteration kernels (ls2d_line.cuh), lengths 108 128 144 162.
#include "ls2d_line.cuh"

namespace mgk {
const Ls2Line* ls2_line_c(int n, int kind) {
  switch (n) {
    case 108: return ls2_pick<108>(kind);
    case 128: return ls2_pick<128>(kind);
    case 144: return ls2_pick<144>(kind);
    case 162: return ls2_pick<162>(kind);
    default: return nullptr;
  }
}
}  // namespace mgk
