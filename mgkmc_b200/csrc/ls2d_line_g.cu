// Instantiations of the 2D iteration kernels (ls2d_line.cuh), lengths 729 768 864.
#include "ls2d_line.cuh"

namespace mgk {
const Ls2Line* ls2_line_g(int n, int kind) {
  switch (n) {
    case 729: return ls2_pick<729>(kind);
    case 768: return ls2_pick<768>(kind);
    case 864: return ls2_pick<864>(kind);
    default: return nullptr;
  }
}
}  // namespace mgk
