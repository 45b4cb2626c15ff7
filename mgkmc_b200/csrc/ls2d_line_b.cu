// Instantiations of the 2D iteration kernels (ls2d_line.cuh), lengths 54 64 72 81 96.
#include "ls2d_line.cuh"

namespace mgk {
const Ls2Line* ls2_line_b(int n, int kind) {
  switch (n) {
    case 54: return ls2_pick<54>(kind);
    case 64: return ls2_pick<64>(kind);
    case 72: return ls2_pick<72>(kind);
    case 81: return ls2_pick<81>(kind);
    case 96: return ls2_pick<96>(kind);
    default: return nullptr;
  }
}
}  // namespace mgk
