// Instantiations of the mixed form's matvec passes (fs3d_mixed_line.cuh), lengths
// 96 108 128 144 162 192 216 243 with the roundings of the CTA-wide passes.
#include "fs3d_mixed_line.cuh"

namespace mgk {
namespace fs32 {
const MixedLine* mixed_line_1c(int n) {
  switch (n) {
    case 96: return mixed_make<96, 1>();
    case 108: return mixed_make<108, 1>();
    case 128: return mixed_make<128, 1>();
    case 144: return mixed_make<144, 1>();
    case 162: return mixed_make<162, 1>();
    case 192: return mixed_make<192, 1>();
    case 216: return mixed_make<216, 1>();
    case 243: return mixed_make<243, 1>();
    default: return nullptr;
  }
}
}  // namespace fs32
}  // namespace mgk
