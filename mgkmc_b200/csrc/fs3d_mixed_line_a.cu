// Instantiations of the mixed form's matvec passes (fs3d_mixed_line.cuh): sides
// 64, 96 and 128 with the roundings of the warp-line kernels.
#include "fs3d_mixed_line.cuh"

namespace mgk {
namespace fs32 {
const MixedLine* mixed_line_0(int n) {
  switch (n) {
    case 64: return mixed_make<64, 0>();
    case 96: return mixed_make<96, 0>();
    case 128: return mixed_make<128, 0>();
    default: return nullptr;
  }
}
}  // namespace fs32
}  // namespace mgk
