// Instantiations of the 2D iteration kernels (ls2d_line.cuh), lengths 486 512 576 648.
#include "ls2d_line.cuh"

namespace mgk {
const Ls2Line* ls2_line_f(int n, int kind) {
  switch (n) {
    case 486: return ls2_pick<486>(kind);
    case 512: return ls2_pick<512>(kind);
    case 576: return ls2_pick<576>(kind);
    case 648: return ls2_pick<648>(kind);
    default: return nullptr;
  }
}
}  // namespace mgk
