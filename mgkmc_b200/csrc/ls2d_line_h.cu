// Instantiations of the 2D iteration kernels (ls2d_line.cuh), lengths 972 1024.
#include "ls2d_line.cuh"

namespace mgk {
const Ls2Line* ls2_line_h(int n, int kind) {
  switch (n) {
    case 972: return ls2_pick<972>(kind);
    case 1024: return ls2_pick<1024>(kind);
    default: return nullptr;
  }
}
}  // namespace mgk
