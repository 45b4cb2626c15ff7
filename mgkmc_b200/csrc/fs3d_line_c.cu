// Instantiations of the finite-strain matvec kernels (fs3d_line.cuh), lengths 144 162 192 216 243 256.
#include "fs3d_line.cuh"

namespace mgk {
const FsLine* fs_line_c(int n) {
  switch (n) {
    case 144: return fs_make<144>();
    case 162: return fs_make<162>();
    case 192: return fs_make<192>();
    case 216: return fs_make<216>();
    case 243: return fs_make<243>();
    case 256: return fs_make<256>();
    default: return nullptr;
  }
}
}  // namespace mgk
