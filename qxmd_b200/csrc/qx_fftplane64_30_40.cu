// FP64 plane and z-column launchers: planes 30x30, 32x32, 36x36, 40x40.
#include "qx_fftplane64_kern.cuh"

namespace qx {
QX_PLANE64_GRID(30, 30)
QX_PLANE64_GRID(32, 32)
QX_PLANE64_GRID(36, 36)
QX_PLANE64_GRID(40, 40)
QX_ZCOLS64_LENGTH(30)
QX_ZCOLS64_LENGTH(32)
QX_ZCOLS64_LENGTH(36)
QX_ZCOLS64_LENGTH(40)
}  // namespace qx
