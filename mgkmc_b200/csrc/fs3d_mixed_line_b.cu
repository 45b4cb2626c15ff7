// Instantiations of the mixed form's matvec passes (fs3d_mixed_line.cuh), lengths
// 24 27 32 36 48 54 64 72 81 with the roundings of the CTA-wide passes.
#include "fs3d_mixed_line.cuh"

namespace mgk {
namespace fs32 {
const MixedLine* mixed_line_1b(int n) {
  switch (n) {
    case 24: return mixed_make<24, 1>();
    case 27: return mixed_make<27, 1>();
    case 32: return mixed_make<32, 1>();
    case 36: return mixed_make<36, 1>();
    case 48: return mixed_make<48, 1>();
    case 54: return mixed_make<54, 1>();
    case 64: return mixed_make<64, 1>();
    case 72: return mixed_make<72, 1>();
    case 81: return mixed_make<81, 1>();
    default: return nullptr;
  }
}
}  // namespace fs32
}  // namespace mgk
