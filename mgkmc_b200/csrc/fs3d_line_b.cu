// Instantiations of the finite-strain matvec kernels (fs3d_line.cuh), lengths 64 72 81 96 108 128.
#include "fs3d_line.cuh"

namespace mgk {
const FsLine* fs_line_b(int n) {
  switch (n) {
    case 64: return fs_make<64>();
    case 72: return fs_make<72>();
    case 81: return fs_make<81>();
    case 96: return fs_make<96>();
    case 108: return fs_make<108>();
    case 128: return fs_make<128>();
    default: return nullptr;
  }
}
}  // namespace mgk
