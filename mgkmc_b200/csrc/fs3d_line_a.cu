// Instantiations of the finite-strain matvec kernels (fs3d_line.cuh), lengths 24 27 32 36 48 54.
#include "fs3d_line.cuh"

namespace mgk {
const FsLine* fs_line_a(int n) {
  switch (n) {
    case 24: return fs_make<24>();
    case 27: return fs_make<27>();
    case 32: return fs_make<32>();
    case 36: return fs_make<36>();
    case 48: return fs_make<48>();
    case 54: return fs_make<54>();
    default: return nullptr;
  }
}
}  // namespace mgk
