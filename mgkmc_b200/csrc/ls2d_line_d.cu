// Instantiations of the 2D iteration kernels (ls2d_line.cuh), lengths 192 216 243 256.
#include "ls2d_line.cuh"

namespace mgk {
const Ls2Line* ls2_line_d(int n, int kind) {
  switch (n) {
    case 192: return ls2_pick<192>(kind);
    case 216: return ls2_pick<216>(kind);
    case 243: return ls2_pick<243>(kind);
    case 256: return ls2_pick<256>(kind);
    default: return nullptr;
  }
}
}  // namespace mgk
