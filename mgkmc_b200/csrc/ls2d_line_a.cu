// Instantiations of the 2D iteration kernels (ls2d_line.cuh), lengths 24 27 32 36 48.
#include "ls2d_line.cuh"

namespace mgk {
const Ls2Line* ls2_line_a(int n, int kind) {
  switch (n) {
    case 24: return ls2_pick<24>(kind);
    case 27: return ls2_pick<27>(kind);
    case 32: return ls2_pick<32>(kind);
    case 36: return ls2_pick<36>(kind);
    case 48: return ls2_pick<48>(kind);
    default: return nullptr;
  }
}
}  // namespace mgk
