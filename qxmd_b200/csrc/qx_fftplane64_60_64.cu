// FP64 plane and z-column launchers: planes 60x60, 64x64.
#include "qx_fftplane64_kern.cuh"

namespace qx {
QX_PLANE64_GRID(60, 60)
QX_PLANE64_GRID(64, 64)
QX_ZCOLS64_LENGTH(60)
QX_ZCOLS64_LENGTH(64)
}  // namespace qx
